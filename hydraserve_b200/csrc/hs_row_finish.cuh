// The counting path after the counting: one CTA turns a row's count table (hs_row_v3.cuh) into its
// sample, in a few phases.  What the phases hand on lives in shared memory, and each phase is a function
// of its own: in one body the values that are alive across it filled the 64 registers twice over,
// and with two CTAs on an SM almost all of L1 is shared memory, so every spilled value was a round
// trip to L2.  What bounds it now is the fetching of instructions a CTA goes through once, and the
// barriers between the passes.  With its count table kept in shared memory and one histogram for all
// cuts, 64 rows of 151,936 with 20 log-probabilities took 75 us instead of 90 (72 now), 1,024 mixed rows of
// 151,936 210 instead of 231 (199 now).
#pragma once

#include "hs_row_v3.cuh"
#include "hs_row_topk.cuh"

namespace hs {

// What a draw asks for when it does not know the token yet: the nth (by ascending id) member of
// the cut's tie group, or of one class.
struct DrawAsk {
  int kind;  // 0 = the token is known (or there is none), 1 = of the group, 2 = of a class
  int token;
  int cell;
  u64 nth, members;
};

struct CountState {
  Ctx3 c;
  hs_row_params P;
  hs_row_out out;        // the row's record, written out in one piece at the end
  KeptSet kept;
  V3Map all_map;         // every token, by score
  u64 q_kept, n_kept, cut_group_cnt;
  long long cut_ties;
  u64 side_best;         // highest side element, (key, ~id); 0 = none
  uint32_t max_key;
  int status, token, scratch;
  Selection sel;         // what select_key found
  DrawAsk ask;           // what the draw left to be found
  Group cut_group;
  bool have_cut_group, tie_split, filled, slot_ok, penalised;
  // from the launch's arguments
  int row, flags, token_draw, s_cap_all, n_scratch;
  int2* s_pair_all;
  int* scratch_busy;
  const float* noise;
  float* scores_out;
  int32_t* tokens_out;
  hs_row_out* out_row;
  ulonglong2* mail_row;
  uint32_t mail_tag;
  int parts;              // CTAs that counted the row; of several, each left a list of its classes
  const uint32_t* lists;  // [parts, kHandedCap]
  const int2* lens;       // [parts]
  unsigned long long* clocks;
};
static_assert(sizeof(CountState) <= kStateBytes, "the state fits its place");
__device__ __forceinline__ CountState& count_state() { return *at_smem<kLayV3.state, CountState>(); }
__device__ __forceinline__ int* count_small() { return at_smem<kLayV3.small, int>(); }
__device__ __forceinline__ void phase_mark(const CountState& S, int slot) {
  if (S.clocks && threadIdx.x == 0) S.clocks[slot] = clock64();
}
// Sets a field of the state (the same value in every thread; visible after the next barrier).
template <class T, class V>
__device__ __forceinline__ void put_state(T& field, V value) {
  if (threadIdx.x == 0) field = (T)value;
}
__device__ __forceinline__ void raise_status(CountState& S, int bits) {
  if (threadIdx.x == 0) S.status |= bits;
}

// Global scratch, for side lists that shared memory does not hold, is kept per RESIDENT CTA: a CTA in
// need claims one of the n_scratch sets (as many as CTAs can be resident, so one is always free),
// starting its search at the pair of its SM, and gives it back at the end.
__device__ bool claim_scratch(CountState& S) {
  if (threadIdx.x == 0) {
    unsigned smid;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
    int got = -1;
#pragma unroll 1
    for (int k = 0; k < 2 * S.n_scratch && got < 0; ++k) {
      const int at = (int)((2u * smid + (unsigned)k) % (unsigned)S.n_scratch);
      if (atomicCAS(&S.scratch_busy[at], 0, 1) == 0) got = at;
    }
    S.scratch = got;
    if (got >= 0) { S.c.s_pair = S.s_pair_all + (size_t)got * S.s_cap_all; S.c.s_cap = S.s_cap_all; }
  }
  __syncthreads();
  return S.scratch >= 0;
}

// ---- selection -------------------------------------------------------------------------------------
// A CTA goes through the chain of selections once per row, so what it costs is first of all the
// fetching of its instructions: one copy of each function, loops that are not unrolled.
__device__ __forceinline__ void hist_add(uint32_t* hist, int b, uint32_t cnt, u64 mass) {
  atomicAdd(hist + b, cnt);
  shared_add_u64(hist + kV3Buckets + b, hist + 2 * kV3Buckets + b, mass);
}
__device__ __forceinline__ u64 hist_mass(const uint32_t* hist, int b) {
  return (u64)hist[kV3Buckets + b] | ((u64)hist[2 * kV3Buckets + b] << 32);
}
// The histogram of count and mass: of every token (side elements one by one, classes with their
// count), or (side_ids) of the kept side elements keyed by ~id.  The thousands of values next to
// zero share a bucket, and would queue up at one address: a warp whose cells all fall into one bucket
// adds them up first.
__device__ __noinline__ void fill_hist(const V3Map map, bool side_ids) {
  CountState& S = count_state();
  Ctx3& c = S.c;
  uint32_t* hist = c.hist();
  const float m = c.m;
#pragma unroll
  for (int b = 0; b < 3 * kV3Buckets / kThreads; ++b) hist[threadIdx.x + b * kThreads] = 0;
  __syncthreads();
  const uint32_t cut_key = S.kept.cut_key;
  for_each_side3(c, [&](int id, float s) {
    const uint32_t key = side_ids ? ~(uint32_t)id : key_of(s);
    if (side_ids && key_of(s) <= cut_key) return;
    if (map.in(key)) hist_add(hist, map.bucket(key), 1u, mass_of(s, m));
  });
  if (!side_ids) {
    for_each_class(c, [&](bool valid, float s, uint32_t n, int) {
      int b;
      if (map.lin) {
        b = map.bucket_of(s);
      } else {
        const uint32_t key = key_of(s);
        valid = valid && map.in(key);
        b = map.bucket(key);
      }
      const u64 w = (u64)n * mass_of(s, m);
      const int first = __reduce_min_sync(0xffffffffu, valid ? b : 0x7fffffff);
      if (__all_sync(0xffffffffu, !valid || b == first)) {
        const uint32_t cnt = __reduce_add_sync(0xffffffffu, valid ? n : 0u);
        const u64 sum = warp_sum_u64(valid ? w : 0ull);
        if (cnt && (threadIdx.x & 31) == 0) hist_add(hist, first, cnt, sum);
      } else if (valid) {
        hist_add(hist, b, n, w);
      }
    });
  }
  __syncthreads();
}

// The key, from the top, at which the running count (by_mass: mass) of the elements reaches
// `target`, with what lies above and at it, in S.sel.  S.filled: the histogram holds all tokens
// under S.all_map (kept up to date).
__device__ __noinline__ void select_key(bool by_mass, bool side_ids, u64 target) {
  CountState& S = count_state();
  Ctx3& c = S.c;
  const int tid = threadIdx.x;
  uint32_t* hist = c.hist();
  V3Map map = S.all_map;
  if (side_ids) map.by_key(~(uint32_t)(c.vocab - 1), 0xffffffffu);
  u64 above = 0;  // of what is counted, above the buckets looked at so far
  if (tid == 0) {
    S.sel.above_cnt = S.sel.above_mass = 0;
    S.sel.target = target;
    S.sel.ok = true;
  }
#pragma unroll 1
  for (int round = 0; round < 8; ++round) {
    if (round > 0 || side_ids || !S.filled) {
      __syncthreads();
      fill_hist(map, side_ids);
      put_state(S.filled, round == 0 && !side_ids);
    }
    if (tid == 0) { c.x()->bcast[7] = 0; *c.gbuf_n() = 0; c.span()[0] = 0xffffffffu; c.span()[1] = 0u; }
    // thread t owns the two buckets 1,023 - 2 t and 1,022 - 2 t
    static_assert(kV3Buckets == 2 * kThreads, "two buckets per thread");
    const int hi = kV3Buckets - 1 - 2 * tid;
    u64 ac, am;  // above this thread's buckets
    {
      const u64 n = (u64)hist[hi] + hist[hi - 1];
      const u64 q = hist_mass(hist, hi) + hist_mass(hist, hi - 1);
      const u64 ia = warp_scan_u64(n), ib = warp_scan_u64(q);
      u64 pa, pb, ta, tb;
      block_warp_prefix2(*c.x(), shfl_u64(ia, 31), shfl_u64(ib, 31), pa, pb, ta, tb);
      ac = pa + ia - n;
      am = pb + ib - q;
    }
    const u64 want = target - above;
#pragma unroll 1
    for (int b = hi; b >= hi - 1; --b) {
      const u64 n = hist[b], q = hist_mass(hist, b);
      const u64 over = by_mass ? am : ac;
      if (over < want && want <= over + (by_mass ? q : n)) {
        c.x()->bcast[0] = (u64)b;
        c.x()->bcast[1] = ac;
        c.x()->bcast[2] = am;
        c.x()->bcast[3] = n;
        c.x()->bcast[4] = q;
        c.x()->bcast[7] = 1;
      }
      ac += n;
      am += q;
    }
    __syncthreads();
    if (c.x()->bcast[7] == 0) {  // nothing reaches the target
      put_state(S.sel.ok, false);
      put_state(S.sel.key, map.klo);
      put_state(S.sel.bin_cnt, 0);
      break;
    }
    const int bucket = (int)c.x()->bcast[0];
    above += by_mass ? c.x()->bcast[2] : c.x()->bcast[1];
    if (tid == 0) {
      S.sel.above_cnt += c.x()->bcast[1];
      S.sel.above_mass += c.x()->bcast[2];
      S.sel.bin_cnt = c.x()->bcast[3];
      S.sel.bin_mass = c.x()->bcast[4];
    }
    phase_mark(S, 22);
    // its members
    {
      const float m = c.m;
      const Scorer sc = c;
      const uint32_t cut_key = S.kept.cut_key;
      auto note = [&](uint32_t key, uint32_t cnt, u64 w) {
        const int slot = atomicAdd(c.gbuf_n(), 1);
        if (slot < kV3ListCap) c.members()[slot] = V3Member{key, cnt, w};
        atomicMin(c.span(), key);
        atomicMax(c.span() + 1, key);
      };
      for_each_side3(c, [&](int id, float s) {
        const uint32_t key = side_ids ? ~(uint32_t)id : key_of(s);
        if (side_ids && key_of(s) <= cut_key) return;
        if (map.in(key) && map.bucket(key) == bucket) note(key, 1u, mass_of(s, m));
      });
      if (!side_ids) {
        locate_cells(c, map, bucket);
        for_located_cells(c, [&](uint32_t n, int cell) {
          const float s = sc.cell_score(cell);
          note(key_of(s), n, (u64)n * mass_of(s, m));
        });
      }
    }
    __syncthreads();
    phase_mark(S, 23);
    const int members = *c.gbuf_n();
    const uint32_t key_lo = c.span()[0], key_hi = c.span()[1];
    if (key_lo == key_hi) { put_state(S.sel.key, key_lo); break; }
    if (members <= kV3ListCap) {
      // each member against all: what lies above its key, and at it
      const u64 still = target - above;
      if (tid < members) {
        const uint32_t mine = c.members()[tid].key;
        u64 oc = 0, om = 0, gc = 0, gm = 0;
#pragma unroll 2
        for (int j = 0; j < members; ++j) {
          const V3Member o = c.members()[j];
          if (o.key > mine) { oc += o.cnt; om += o.w; }
          if (o.key == mine) { gc += o.cnt; gm += o.w; }
        }
        const u64 over = by_mass ? om : oc;
        if (over < still && still <= over + (by_mass ? gm : gc)) {  // (members of one key write the same)
          c.x()->bcast[0] = mine;
          c.x()->bcast[1] = oc; c.x()->bcast[2] = om; c.x()->bcast[3] = gc; c.x()->bcast[4] = gm;
        }
      }
      __syncthreads();
      if (tid == 0) {
        S.sel.key = (uint32_t)c.x()->bcast[0];
        S.sel.above_cnt += c.x()->bcast[1];
        S.sel.above_mass += c.x()->bcast[2];
        S.sel.bin_cnt = c.x()->bcast[3];
        S.sel.bin_mass = c.x()->bcast[4];
      }
      break;
    }
    map.by_key(key_lo, key_hi);
    __syncthreads();
  }
  __syncthreads();
}

// Count and mass of all tokens with key >= lo_key, in S.sel.total_cnt / total_mass.
__device__ __noinline__ void totals3(uint32_t lo_key) {
  CountState& S = count_state();
  Ctx3& c = S.c;
  u64 a = 0, b = 0;
  if (S.filled && lo_key == 0u) {
#pragma unroll
    for (int u = 0; u < kV3Buckets / kThreads; ++u) {
      const int i = threadIdx.x + u * kThreads;
      a += c.hist()[i];
      b += hist_mass(c.hist(), i);
    }
  } else {
    const float m = c.m;
    for_each_side3(c, [&](int, float s) {
      if (key_of(s) >= lo_key) { ++a; b += mass_of(s, m); }
    });
    for_each_class(c, [&](bool valid, float s, uint32_t n, int) {
      if (valid && key_of(s) >= lo_key) { a += n; b += (u64)n * mass_of(s, m); }
    });
  }
  block_sum2(*c.x(), a, b);
  put_state(S.sel.total_cnt, a);
  put_state(S.sel.total_mass, b);
  __syncthreads();
}

// The side list (tokens held three times or more, values outside the bin window), the row's maximum
// and minimum, and every token's count and mass in one histogram over the scores.  False: no scratch.
__device__ __noinline__ bool phase_histogram() {
  CountState& S = count_state();
  Ctx3& c = S.c;
  int* small = count_small();
  const int tid = threadIdx.x, lane = tid & 31;
  const bool penalised = S.penalised;
  // (id, count, value) of a token held three times or more are three dependent reads: thread t
  // starts the chain for list entry t here and takes one step of it at each stop below
  int n_heavy = 0, hv_q = -1;
  const int cap = c.pool.unique_cap;
  const int32_t* heavy = c.pool.heavy + (size_t)max(c.slot, 0) * cap;
  const int2* pairs = c.pool.pairs + (size_t)max(c.slot, 0) * cap;
  if (penalised) {
    n_heavy = load_now_s32(c.pool.n_heavy + c.slot);
    if (tid < cap) hv_q = load_now_s32(heavy + tid);
  }
  // ---- highest and lowest non-empty cell of each count class: scores grow with the bin inside one
#pragma unroll 1
  for (int k = 0; k < (penalised ? 3 : 1); ++k) {  // (without penalties there is one count class)
    uint32_t bits = 0;
#pragma unroll
    for (int u = 0; u < kPerClass; ++u) bits |= (c.tab()[tid + (k * kPerClass + u) * kThreads] ? 1u : 0u) << u;
    const uint32_t t = __reduce_max_sync(0xffffffffu, bits ? (uint32_t)(tid + (k * kPerClass + 31 - __clz(bits)) * kThreads) + 1u : 0u);
    const uint32_t l = __reduce_min_sync(0xffffffffu, bits ? (uint32_t)(tid + (k * kPerClass + __ffs(bits) - 1) * kThreads) : 0xffffffffu);
    if (lane == 0) {
      if (t) atomicMax(reinterpret_cast<unsigned*>(small) + 16 + k, t);
      if (l != 0xffffffffu) atomicMin(reinterpret_cast<unsigned*>(small) + 19 + k, l);
    }
  }
  // (more often-repeated tokens than the side list holds: the general kernel's row)
  if (n_heavy > min(cap, S.s_cap_all)) raise_status(S, 4);
  n_heavy = min(n_heavy, min(cap, S.s_cap_all));
  int2 hv_pair = make_int2(-1, 0);
  if (tid < n_heavy && hv_q >= 0 && hv_q < cap) hv_pair = load_now_int2(pairs + hv_q);  // (id, count)
  const int n_rare = small[1];
  if (n_rare > kV3RareCap || n_heavy + kV3RareCap > kV3SideShared) {
    if (!claim_scratch(S)) return false;
  }
  // ---- the side list.  It is walked by every selection, so it lives in shared memory when it fits.
  {
    const Ctx3 k = c;  // (what scoring needs, in registers)
    u64 side_best = 0;
    uint32_t side_worst = 0xffffffffu;  // this thread's lowest side key
    auto put = [&](int slot, int id, float s) {
      if (slot >= k.s_cap) return;  // (reported below, from the counts, by every thread alike)
      k.s_pair[slot] = make_int2(id, __float_as_int(s));
      const u64 packed = ((u64)key_of(s) << 32) | (uint32_t)(~(uint32_t)id);
      side_best = packed > side_best ? packed : side_best;
      side_worst = min(side_worst, key_of(s));
    };
#pragma unroll 1
    for (int j = tid; j < n_heavy; j += kThreads) {
      if (j != tid) {  // (the first entry's reads were started early)
        const int q = heavy[j];
        hv_pair = q >= 0 && q < cap ? pairs[q] : make_int2(-1, 0);
      }
      if (hv_pair.x < 0 || hv_pair.x >= k.vocab) { if (j < k.s_cap) k.s_pair[j] = make_int2(-1, 0); }
      else put(j, hv_pair.x, k.score_of(k.logits[hv_pair.x], hv_pair.y));
    }
    int n_s = n_heavy + n_rare;
    if (n_rare <= kV3RareCap) {
      const int2* rare = c.rare();
#pragma unroll 1
      for (int t = tid; t < n_rare; t += kThreads) {
        const int2 e = rare[t];
        put(n_heavy + t, e.x, k.score_of((uint32_t)e.y & 0xffffu, (e.y >> 16) & 3));
      }
    } else {
      // too many to remember: sweep the row again for out-of-window values
#pragma unroll 1
      for (int id = tid; id < k.vocab; id += kThreads) {
        const uint32_t raw = k.logits[id];
        const int cc = k.class_of(id);
        if (cc == 3 || v3_bin_of_raw(raw) >= 0) continue;
        put(n_heavy + atomicAdd(small + 2, 1), id, k.score_of(raw, cc));
      }
      __syncthreads();
      n_s = n_heavy + small[2];
    }
    // more than the list holds: the row is reported for the general kernel (from the counts, not by
    // the thread whose token found no room)
    if (n_s > k.s_cap) raise_status(S, 4);
    put_state(c.n_s, min(n_s, k.s_cap));
    const u64 sb = warp_max_u64(side_best);
    const uint32_t sl = __reduce_min_sync(0xffffffffu, side_worst);
    if (lane == 0) {
      if (sb) atomicMax(&c.x()->bcast[5], sb);
      if (sl != 0xffffffffu) atomicMin(reinterpret_cast<unsigned*>(small) + 22, sl);
    }
  }
  __syncthreads();
  phase_mark(S, 11);
  // ---- row maximum and minimum: the scores of six cells, one per lane, and the side list's ends
  {
    const bool top = lane < 3;
    const uint32_t mark_at = reinterpret_cast<unsigned*>(small)[(top ? 16 : 19) + lane % 3];
    const bool valid = lane < 6 && (top ? mark_at != 0u : mark_at != 0xffffffffu);
    uint32_t key = 0;
    if (valid) key = key_of(c.cell_score(top ? (int)mark_at - 1 : (int)mark_at));
    const u64 side_best = c.x()->bcast[5];
    const uint32_t max_key = max(__reduce_max_sync(0xffffffffu, valid && top ? key : 0u), (uint32_t)(side_best >> 32));
    const uint32_t min_key = min(__reduce_min_sync(0xffffffffu, valid && !top ? key : 0xffffffffu), reinterpret_cast<unsigned*>(small)[22]);
    if (tid == 0) {
      S.side_best = side_best;
      S.max_key = max_key;
      c.m = score_of(max_key);
      V3Map map;
      map.by_score(score_of(min_key), score_of(max_key));
      S.all_map = map;
    }
  }
  __syncthreads();
  phase_mark(S, 2);
  // ---- the histogram (in the place of the rare tokens and set-aside chunks, which have served)
  if (!c.greedy || S.P.n_logprobs >= 0) {
    fill_hist(S.all_map, false);
    put_state(S.filled, true);
    __syncthreads();
  }
  phase_mark(S, 3);
  return true;
}

// Top-k, min-p and top-p.  What a cut keeps lies at the top, so every cut is looked for among all tokens.
__device__ __noinline__ void phase_cuts() {
  CountState& S = count_state();
  Ctx3& c = S.c;
  const hs_row_params& P = S.P;
  const int tid = threadIdx.x;
  uint32_t cut_key = 0;
  u64 cnt = 0, mass = 0;
  bool have_totals = false;
  if (P.top_k > 0 && P.top_k < c.vocab) {
    select_key(false, false, (u64)P.top_k);
    if (!S.sel.ok) raise_status(S, 1);
    cut_key = S.sel.key;
    cnt = S.sel.above_cnt + S.sel.bin_cnt;
    mass = S.sel.above_mass + S.sel.bin_mass;
    have_totals = S.sel.ok;
    put_state(S.out.n_after_topk, cnt);
    put_state(S.cut_group_cnt, S.sel.bin_cnt);
  }
  phase_mark(S, 4);
  if (P.min_p > 0.0f) {
    if (!have_totals) { totals3(cut_key); cnt = S.sel.total_cnt; mass = S.sel.total_mass; have_totals = true; }
    const float z1 = mass_to_float(mass), m = c.m;
    const float thr = __fmul_rn(__fdiv_rn(1.0f, z1), P.min_p);
    uint32_t lowest = 0xffffffffu;
    auto consider = [&](float s) {
      const uint32_t k = key_of(s);
      if (k >= cut_key && k < lowest && !(__fdiv_rn(expf(s - m), z1) < thr)) lowest = k;
    };
    // Of the cells, only those that come near the line: a token passes from m + log(min_p) on, give or
    // take the roundings of exp and of the quotients, parts in a million.  (All of them, when the threshold is
    // no normal number: a subnormal one is off by any share of itself, everything passes 0, and a maximum of
    // infinity leaves no line.)
    const float floor = __fadd_rd(__fadd_rd(m, logf(P.min_p)), -0.01f);
    const bool line = thr >= 1.17549435e-38f && thr < INFINITY && floor > -3.0e38f;
    V3Map near_line;
    near_line.by_key(line ? key_of(floor) : 0u, 0xffffffffu);
    locate_cells(c, near_line, 0);
    const Scorer sc = c;
#pragma unroll 1
    for (int k = 0; k < 3; ++k) {
#pragma unroll 1
      for (int cell = c.range()[k] + tid; cell < c.ends()[k]; cell += kThreads)
        if (c.tab()[cell]) consider(sc.bin_score(cell - k * kV3Bins, k));
    }
    for_each_side3(c, [&](int, float s) { consider(s); });
    lowest = ~block_max_u32(*c.x(), ~lowest);
    if (lowest != 0xffffffffu && lowest > cut_key) {
      cut_key = lowest;
      have_totals = false;
    }
  }
  phase_mark(S, 5);
  if (!have_totals) { totals3(cut_key); cnt = S.sel.total_cnt; mass = S.sel.total_mass; }
  put_state(S.out.n_after_minp, cnt);
  if (P.top_p < 1.0f) {
    if (mass > 0) {
      // (double precision, slow: the lanes of one warp try neighbouring candidates at once)
      if (tid < 32) {
        const u64 t = top_p_target_warp(mass, P.top_p);
        if (tid == 0) c.x()->bcast[6] = t;
      }
      __syncthreads();
      phase_mark(S, 20);
      select_key(true, false, c.x()->bcast[6]);
      phase_mark(S, 21);
    }
    if (mass > 0 && S.sel.ok && S.sel.bin_cnt > 0) {
      const u64 qv = S.sel.bin_mass / S.sel.bin_cnt;  // every token at the cut key has the same mass
      u64 t = S.sel.bin_cnt;
      if (qv > 0) {
        const u64 want = S.sel.target - S.sel.above_mass;
        t = (want + qv - 1) / qv;
        if (t < 1) t = 1;
        if (t > S.sel.bin_cnt) t = S.sel.bin_cnt;
      }
      cut_key = S.sel.key;
      cnt = S.sel.above_cnt + t;
      mass = S.sel.above_mass + t * qv;
      put_state(S.cut_ties, (long long)t);
      put_state(S.cut_group_cnt, S.sel.bin_cnt);
      put_state(S.tie_split, t < S.sel.bin_cnt);
    } else {
      raise_status(S, 1);
    }
  }
  __syncthreads();
  put_state(S.kept.cut_key, cut_key);
  put_state(S.n_kept, cnt);
  put_state(S.q_kept, mass);
  __syncthreads();
  phase_mark(S, 6);
}

__device__ __forceinline__ void need_cut_group(CountState& S) {
  if (S.have_cut_group) return;
  const Group g = find_group(S.c, S.kept.cut_key);
  put_state(S.cut_group, g);
  put_state(S.have_cut_group, true);
  __syncthreads();
}
// The highest id of the cut's tie group that is kept, when top-p split the group.
__device__ __noinline__ void need_tie_limit() {
  CountState& S = count_state();
  if (!S.tie_split || S.kept.tie_limit != 0x7fffffff) return;
  need_cut_group(S);
  const int limit = nth_in_group(S.c, S.cut_group, (u64)S.cut_ties);
  __syncthreads();
  put_state(S.kept.tie_limit, limit);
  __syncthreads();
}

// The draw by classes: inverse CDF over exact integer masses in the order: classes above the cut, the
// tie group at the cut (its lowest ids), side elements above the cut (by id).
__device__ __noinline__ void draw_by_classes(uint64_t seed) {
  CountState& S = count_state();
  Ctx3& c = S.c;
  const int tid = threadIdx.x;
  const uint32_t cut_key = S.kept.cut_key;
  const float m = c.m;
  u64 target;
  {
    const Philox4 r = philox4x32_10(0u, 0u, 0u, 0u, (uint32_t)seed, (uint32_t)(seed >> 32));
    target = __umul64hi(((u64)r.v[0] << 32) | r.v[1], S.q_kept);
  }
  // Classes above the cut in this order: the non-empty cells t, t + kThreads, ... of every t in
  // turn make a list, and its entries j, j + kThreads, ... are chunk j.  (Any fixed order
  // would do; the counts alone decide it.)  A thread adds its cells' masses to their chunks.
  // Only the cells above the cut weigh anything: the others are passed over by their number.  (Bound by the
  // instructions per cell, of which scores and exponentials are most: over all cells this pass took 14.9 thousand
  // cycles a row with top_p in a batch of 1,024 mixed rows, 10.8 this way, the one for min_p above 11.9 and 9.0.)
  const uint32_t* tab = c.tab();
  {
    V3Map at_cut;
    at_cut.by_key(cut_key, cut_key);
    locate_cells(c, at_cut, 0);  // (range()[3 + k]: the first cell of count class k above the cut)
  }
  int mine = 0;
#pragma unroll 1
  for (int k = 0; k < 3; ++k) {
    if (c.ends()[k] == 0) continue;
#pragma unroll
    for (int u = 0; u < kPerClass; ++u) mine += tab[tid + (k * kPerClass + u) * kThreads] ? 1 : 0;
  }
  uint32_t* chunks = reinterpret_cast<uint32_t*>(c.members());  // [2][kThreads]: mass, low and high words
  static_assert(2 * kThreads * sizeof(uint32_t) <= sizeof(V3Member) * kV3ListCap + sizeof(int) * kV3TieCap, "the chunks fit the members' place");
#pragma unroll
  for (int l = 0; l < 2; ++l) chunks[tid + l * kThreads] = 0;
  int n_cl;
  const int list_at = block_place(count_small() + 48, mine, n_cl);
  {
    const Scorer sc = c;
    int from = list_at;  // (a thread's cells come in the order of the list)
#pragma unroll 1
    for (int k = 0; k < 3; ++k) {
      if (c.ends()[k] == 0) continue;
      uint32_t bits = 0;
#pragma unroll
      for (int u = 0; u < kPerClass; ++u) bits |= (tab[tid + (k * kPerClass + u) * kThreads] ? 1u : 0u) << u;
      // (this thread's first cell at or behind the first one above the cut)
      const int u0 = max(0, c.range()[3 + k] - k * kV3Bins - tid + kThreads - 1) / kThreads;
      uint32_t left = u0 < kPerClass ? bits & (0xffffffffu << u0) : 0u;
#pragma unroll 1
      while (left) {
        const int u = __ffs(left) - 1;
        left &= left - 1u;
        const int cell = tid + (k * kPerClass + u) * kThreads;
        const u64 w = (u64)tab[cell] * mass_of(sc.bin_score(cell - k * kV3Bins, k), m);
        uint32_t* dst = chunks + ((from + __popc(bits & ((1u << u) - 1u))) & (kThreads - 1));
        shared_add_u64(dst, dst + kThreads, w);
      }
      from += __popc(bits);
    }
  }
  __syncthreads();
  const u64 chunk = (u64)chunks[tid] | ((u64)chunks[tid + kThreads] << 32);
  const u64 incl = warp_scan_u64(chunk);
  u64 pre, pre_unused, q_cells, tot_unused;
  block_warp_prefix2(*c.x(), shfl_u64(incl, 31), 0, pre, pre_unused, q_cells, tot_unused);
  phase_mark(S, 12);
  if (target < q_cells) {
    // the chunk that holds the target, its cells in order (a thread has at most one of them:
    // its entries of the list are fewer than kThreads and lie side by side), then the cell
    int* cells = c.list();
    constexpr int kMostCells = kCells / kThreads;
    if (tid < kMostCells) cells[tid] = -1;
    if (tid == 0) c.x()->bcast[5] = 0;
    const u64 from = pre + incl - chunk;
    if (from <= target && target < from + chunk) { c.x()->bcast[0] = (u64)tid; c.x()->bcast[1] = from; }
    __syncthreads();
    {
      int skip = ((int)c.x()->bcast[0] - list_at) & (kThreads - 1);
      if (skip < mine) {
        const int slot = (list_at + skip) / kThreads;
        int cell = tid;
#pragma unroll 1
        while (tab[cell] == 0u || skip-- > 0) cell += kThreads;
        cells[slot] = cell;
      }
    }
    __syncthreads();
    if (tid < 32) {
      u64 run = c.x()->bcast[1];
#pragma unroll 1
      for (int base = 0; base < kMostCells; base += 32) {
        const int cell = base + tid < kMostCells ? cells[base + tid] : -1;
        u64 q = 0, w = 0;
        if (cell >= 0) {
          const uint32_t key = key_of(c.cell_score(cell));
          if (key > cut_key) { q = mass_of(score_of(key), m); w = (u64)tab[cell] * q; }
        }
        const u64 in = warp_scan_u64(w);
        if (w && run + in - w <= target && target < run + in) {
          c.x()->bcast[3] = tab[cell];
          c.x()->bcast[4] = (target - (run + in - w)) / q + 1;
          c.x()->bcast[5] = (u64)cell + 1;
        }
        run += shfl_u64(in, 31);
      }
    }
    __syncthreads();
    const int cell = (int)c.x()->bcast[5] - 1;
    put_state(S.ask, DrawAsk{cell >= 0 ? 2 : 0, -1, cell, c.x()->bcast[4], c.x()->bcast[3]});
    return;
  }
  // the group at the cut key: cut_ties members when top-p split it, else all of them
  u64 group_kept = (u64)S.cut_ties;
  if (S.cut_ties < 0) {
    // cut by top-k / min-p / nothing: everything at the cut key is kept; count it
    u64 gc = 0, gm = 0;
    V3Map at_key;
    at_key.by_key(cut_key, cut_key);
    locate_cells(c, at_key, 0);
    for_located_cells(c, [&](uint32_t n, int) { gc += n; });
    for_each_side3(c, [&](int, float s) { if (key_of(s) == cut_key) gc += 1; });
    block_sum2(*c.x(), gc, gm);
    group_kept = gc;
  }
  const u64 q_cut = mass_of(score_of(cut_key), m);
  const u64 q_group = group_kept * q_cut;
  if (target < q_cells + q_group) {
    put_state(S.ask, DrawAsk{1, -1, -1, q_cut ? (target - q_cells) / q_cut + 1 : 1ull, 0ull});
    return;
  }
  select_key(true, true, target - q_cells - q_group + 1);
  put_state(S.ask, DrawAsk{0, S.sel.ok ? (int)(~S.sel.key) : -1, -1, 0ull, 0ull});
}

// Token id of the n-th (1-based, ascending id) member of one class, of at most kV3ScanCap tokens, of a row
// that several CTAs counted (-1: there is none).  The parts are ranges of the row in order, and each left
// a list of its classes with their counts, in the order of the cells: a warp looks the class up in
// each list, 32 entries at a time, the counts name the part, and that range alone is scanned.  (The loose
// tokens belong to the last part, those ahead of the first chunk too.)  Bound by the latency of three or
// four reads and of the range's: from the cuts to the token 31.8 thousand cycles with a scan of the row, 26.7 this
// way (one row of 248,320 in seven parts, a call 64.1 and 61.7 us), 29.3 and 26.2 (37 rows of 151,936 in four).
__device__ __noinline__ int nth_in_parts(int cell, u64 n) {
  CountState& S = count_state();
  Ctx3& c = S.c;
  int* small = count_small();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cc = cell / kV3Bins, parts = S.parts;
  const uint32_t raw = v3_raw_of_bin(cell - cc * kV3Bins);
  uint32_t ahead = 0;  // members ahead of the first chunk
  if (c.head())
    ahead = __ballot_sync(0xffffffffu, lane < c.head() && (uint32_t)c.logits[lane] == raw && c.class_of(lane) == cc);
  if (n <= (u64)__popc(ahead)) return (int)__fns(ahead, 0, (int)n);
  __syncthreads();
  if (warp < parts) {
    const uint32_t* list = S.lists + (size_t)warp * kHandedCap;
    const int len = __ldcg(S.lens + warp).x;
    int lo = 0, hi = len;
#pragma unroll 1
    while (lo < hi) {
      const int step = (hi - lo + 31) >> 5;
      const int t = lo + (lane + 1) * step - 1;
      const bool pass = t >= hi || (int)(__ldcg(list + t) & 0x7fffu) >= cell;
      const uint32_t votes = __ballot_sync(0xffffffffu, pass);
      if (votes == 0) { lo = hi; break; }
      const int first = __ffs(votes) - 1;
      hi = min(lo + (first + 1) * step - 1, hi);
      lo = lo + first * step;
    }
    if (lane == 0) {
      const uint32_t e = lo < len ? __ldcg(list + lo) : 0u;
      small[48 + warp] = e && (int)(e & 0x7fffu) == cell ? (int)(e >> 15) : 0;
    }
  }
  if (threadIdx.x == 0) *c.gbuf_n() = 0;
  __syncthreads();
  int before = __popc(ahead), in_part = 0, g = 0;
#pragma unroll 1
  for (; g < parts; ++g) {
    in_part = small[48 + g] - (g == parts - 1 ? __popc(ahead) : 0);
    if (n <= (u64)(before + in_part)) break;
    before += in_part;
  }
  if (g == parts) return -1;
  const int per = chunks_per_part(c.n8(), parts), first = min(g * per, c.n8());
  // (the part as a row of its own, its ids counted from `from`; a last part without a chunk, which need not start
  // on a whole word of classes, has the loose tokens alone)
  ScanArgs a = scan_args(c);
  a.n8 = min(per, c.n8() - first);
  const int from = a.n8 ? 8 * first : 0;
  a.logits += from;
  if (a.cls) a.cls += from / 16;
  a.head += 8 * first - from;
  a.vocab = g < parts - 1 ? a.head + 8 * a.n8 : c.vocab - from;
  a.front = 0;
  scan_members<true>(a, raw, kNoRaw, kNoRaw, cc, (int)n - before, in_part);
  const u64 hit = c.x()->bcast[6];
  __syncthreads();
  return hit ? from + (int)hit - 1 : -1;
}

// Finds what a draw asks for: its own function, for the registers of the scan.
__device__ __noinline__ int phase_find() {
  CountState& S = count_state();
  Ctx3& c = S.c;
  const DrawAsk ask = S.ask;
  if (ask.kind == 1) {
    need_cut_group(S);
    return nth_in_group(c, S.cut_group, ask.nth);  // the kept members are the lowest ids
  }
  // a uniformly chosen member of ONE class (not of other classes that share its key):
  // large classes by rejection (about vocab / members scattered probes, which a lone CTA
  // issues slowly), classes of up to kV3RejectMin tokens by one scan of the row
  int token = -1;
  const int cell = ask.cell;
  if (ask.members > (u64)kV3RejectMin) {
    const u64 per_round = ((u64)c.vocab + ask.members - 1) / ask.members;  // probes for ~63 % success
    const int trials = (int)min((u64)kRandomTrials, max(1ull, (per_round + kThreads - 1) / kThreads));
    // a class the scan can hold gets a few rounds, then the scan; a larger one many
    token = random_in_class(c, cell, trials, S.P.seed, ask.members <= (u64)kV3ScanCap ? 4 : 32);
  }
  if (token >= 0) return token;
  if (S.parts > 1 && ask.members <= (u64)kV3ScanCap && (token = nth_in_parts(cell, ask.nth)) >= 0) return token;
  // (no key: no other member can match)
  const Group only{0xffffffffu, cell < kV3Bins ? cell : -1, cell >= kV3Bins && cell < 2 * kV3Bins ? cell : -1,
                   cell >= 2 * kV3Bins ? cell : -1};
  return nth_in_group(c, only, ask.nth);
}

// The token under the reference's own draws: arg max of fl(fl(e / z) / noise) over the kept set, lowest
// id on ties.
__device__ __noinline__ int draw_from_noise() {
  CountState& S = count_state();
  Ctx3& c = S.c;
  need_tie_limit();
  const KeptSet kept = S.kept;
  const float zf = mass_to_float(S.q_kept), m = c.m;
  const float* noise_row = S.noise + (size_t)S.row * c.vocab;
  u64 best = 0;
#pragma unroll 1
  for (int id = threadIdx.x; id < c.vocab; id += kThreads) {
    const float s = c.element_score(id, c.logits[id], c.class_of(id));
    if (!kept.has(key_of(s), id)) continue;
    const float p = __fdiv_rn(expf(s - m), zf);
    const float ratio = __fdiv_rn(p, noise_row[id]);
    const u64 packed = ((u64)__float_as_uint(ratio) << 32) | (uint32_t)(~(uint32_t)id);
    best = packed > best ? packed : best;
  }
  best = block_max_u64(*c.x(), best);
  return (int)(~(uint32_t)(best & 0xffffffffu));
}

// The draw: the token, or what is left to be found of it, in S.ask.
__device__ __noinline__ void phase_draw() {
  CountState& S = count_state();
  Ctx3& c = S.c;
  const uint64_t seed = S.P.seed;
  if (S.q_kept == 0 || S.noise) {
    // (nothing has any mass: no token, reported by the caller)
    const int token = S.q_kept == 0 ? -1 : draw_from_noise();
    put_state(S.ask, DrawAsk{0, token, -1, 0ull, 0ull});
    return;
  }
  // Near-flat rows: rejection on tokens, when one round is all but sure to accept.
  const float q = mass_to_float(S.q_kept);
  if (S.token_draw && q * (float)(kTokenTrials * kThreads) >= 4.0f * (float)c.vocab) {
    bool group_hit;
    // (a sixteenth of the trials accepted on average: one per thread is plenty)
    const int trials = q * 16.0f >= (float)c.vocab ? 1 : kTokenTrials;
    const u64 ties = S.cut_ties > 0 ? (u64)S.cut_ties : 0ull;
    const int t = draw_by_token_rejection(c, S.kept, S.tie_split, ties, S.cut_group_cnt, seed, 4, trials, group_hit);
    if (t >= 0) {
      u64 nth = 0;
      if (group_hit) {
        // one of the kept members of the group the cut splits: its lowest ids
        const Philox4 r = philox4x32_10(0u, 0u, 0u, 4u, (uint32_t)seed, (uint32_t)(seed >> 32));
        nth = 1 + __umul64hi(((u64)r.v[0] << 32) | r.v[1], ties);
      }
      put_state(S.ask, DrawAsk{group_hit ? 1 : 0, t, -1, nth, 0ull});
      return;
    }
  }
  draw_by_classes(seed);
}

// The tokens of the row at or above `key`: those above it into the gather buffer, with their keys,
// those at it into the list of ids (at most kV3TieCap are kept) with the lowest of them in *low_id.
// Side elements come from the side list, the rest from one walk of the row against per-class raw
// thresholds.
__device__ __noinline__ void collect_at_or_above(uint32_t key, int* low_id) {
  CountState& S = count_state();
  Ctx3& c = S.c;
  int* small = count_small();
  int* tie_n = small + 26;
  if (threadIdx.x == 0) { *c.gbuf_n() = 0; *tie_n = 0; *low_id = 0x7fffffff; }
  __syncthreads();
  auto take = [&](uint32_t k, int id) {
    if (k > key) {
      const int slot = atomicAdd(c.gbuf_n(), 1);
      if (slot < kV3ListCap) c.gbuf()[slot] = V3Entry{k, id};
    } else if (k == key) {
      const int slot = atomicAdd(tie_n, 1);
      if (slot < kV3TieCap) c.list()[slot] = id;
      atomicMin(low_id, id);
    }
  };
  for_each_side3(c, [&](int id, float s) { take(key_of(s), id); });
  CandCtx bound_ctx{nullptr, nullptr, nullptr, nullptr, small + 8, nullptr};
  cand_thresholds(c, bound_ctx, key);  // (ends with a barrier)
  const Scorer sc = c;
  stream_at_or_above(c, bound_ctx.thr, [&](int id, uint32_t raw, int cc) {
    if (v3_bin_of_raw(raw) < 0) return;  // outside the bin window: a side element, taken above
    take(key_of(sc.score_of(raw, cc)), id);
  });
  __syncthreads();
}

// Arg max with penalties: the lowest id among the tokens whose score key is the maximum.
__device__ __noinline__ void phase_greedy() {
  CountState& S = count_state();
  int* low_id = count_small() + 3;
  collect_at_or_above(S.max_key, low_id);
  int token = *low_id;
  if (token == 0x7fffffff) { token = S.side_best ? (int)(~(uint32_t)(S.side_best & 0xffffffffu)) : 0; raise_status(S, 1); }
  put_state(S.token, token);
  if (S.P.n_logprobs >= 0) {
    totals3(0u);
    put_state(S.q_kept, S.sel.total_mass);
  }
  __syncthreads();
}

// Appends the `need` lowest ids of a large tie group to the top-N tokens.
__device__ __noinline__ void emit_lowest_of_group(Ctx3& c, uint32_t key, int need) {
  const int have = *c.gbuf_n();  // (the walk below counts in the same place)
  const Group g = find_group(c, key);
  const int last_id = nth_in_large_group(c, g, (u64)need);
  if (threadIdx.x == 0) *c.gbuf_n() = have;
  __syncthreads();
  emit_group_upto(c, g, last_id == 0x7fffffff ? -1 : last_id);
}

// Log-probabilities: of the token, and of the N highest kept ones.
__device__ __noinline__ void phase_logprobs() {
  CountState& S = count_state();
  Ctx3& c = S.c;
  int* small = count_small();
  const int tid = threadIdx.x;
  if (tid == 0) {
    S.out.log_z = (float)(log((double)S.q_kept) - (double)kMassShift * 0.6931471805599453);
    const int token = S.token;
    if (token >= 0 && token < c.vocab)
      S.out.logprob = (c.element_score(token, c.logits[token], c.class_of(token)) - c.m) - S.out.log_z;
  }
  int n_want = min(S.P.n_logprobs, c.vocab);
  if ((u64)n_want > S.n_kept) n_want = (int)S.n_kept;
  if (n_want > 0) {
    // (the kept tokens are the highest: the N highest of them are the N highest of all)
    select_key(false, false, (u64)n_want);
    if (S.sel.ok) {
      const int need = n_want - (int)S.sel.above_cnt;  // lowest ids of the group at the N-th key
      const uint32_t nth_key = S.sel.key;
      phase_mark(S, 16);
      collect_at_or_above(nth_key, small + 3);
      phase_mark(S, 17);
      int* tie_ids = c.list();
      int* gbuf_n = c.gbuf_n();
      V3Entry* gbuf = c.gbuf();
      if (need > 0) {
        const int n_tie = small[26];
        if (n_tie <= kV3TieCap) {
          // the `need` lowest ids of the group: each id counts the ids below it
#pragma unroll 1
          for (int t = tid; t < n_tie; t += kThreads) {
            const int mine = tie_ids[t];
            int below = 0;
#pragma unroll 4
            for (int j = 0; j < n_tie; ++j) below += tie_ids[j] < mine ? 1 : 0;
            if (below < need) {
              const int slot = atomicAdd(gbuf_n, 1);
              if (slot < kV3ListCap) gbuf[slot] = V3Entry{nth_key, mine};
            }
          }
        } else {
          emit_lowest_of_group(c, nth_key, need);
        }
      }
      __syncthreads();
      if (tid < 32) {
        const int n = min(*gbuf_n, HS_MAX_LOGPROBS);
        uint32_t kv = 0;
        int id = 0x7fffffff;
        if (tid < n) { kv = gbuf[tid].key; id = gbuf[tid].id; }
        int pos = 0;
#pragma unroll 1
        for (int j = 0; j < n; ++j) {
          const uint32_t kj = __shfl_sync(0xffffffffu, kv, j);
          const int idj = __shfl_sync(0xffffffffu, id, j);
          if (kj > kv || (kj == kv && idj < id)) ++pos;
        }
        const float log_z = S.out.log_z;
        if (tid < n) {
          S.out.top_ids[pos] = id;
          S.out.top_logprobs[pos] = (score_of(kv) - c.m) - log_z;
        }
        if (tid == 0 && n != n_want) S.status |= 8;
      }
    } else {
      n_want = 0;
      raise_status(S, 1);
    }
  }
  put_state(S.out.n_top, n_want);
  __syncthreads();
  phase_mark(S, 8);
}

// Gives a claimed set of global scratch back.
__device__ __forceinline__ void release_scratch(CountState& S) {
  if (S.scratch >= 0 && threadIdx.x == 0) { __threadfence(); atomicExch(&S.scratch_busy[S.scratch], 0); }
}

// A candidate row whose list overflowed while it was streamed.  Whether one does depends on how many
// CTAs share the row, and so on the batch around it, and the token a seed names must not: with the
// tokens counted, the k-th highest score is known exactly, and when the k highest and the ties of
// the last fit a list after all, they are listed (in the count table's place, which has served) and
// the row is finished like any other of its kind.  False: they do not fit, or the row goes to the
// general kernel.  Bound by one more walk of the row, in the place of the draw's.
__device__ __noinline__ bool finish_listed_row() {
  CountState& S = count_state();
  Ctx3& c = S.c;
  if (S.status & 4) return false;
  select_key(false, false, (u64)S.P.top_k);
  if (!S.sel.ok || S.sel.above_cnt + S.sel.bin_cnt > (u64)kCandCap) return false;
  static_assert(2 * kCandCap * sizeof(u64) <= sizeof(uint32_t) * kCells, "list and masses fit the count table's place");
  u64* list = at_smem<kLayV3.tab, u64>();
  const uint32_t key = S.sel.key;
  if (threadIdx.x == 0) *c.gbuf_n() = 0;
  __syncthreads();
  auto take = [&](uint32_t k, int id) {
    if (k < key) return;
    const int slot = atomicAdd(c.gbuf_n(), 1);
    if (slot < kCandCap) list[slot] = cand_pack(k, id);
  };
  for_each_side3(c, [&](int id, float s) { take(key_of(s), id); });
  CandCtx L{list, nullptr, nullptr, nullptr, count_small() + 8, nullptr};
  cand_thresholds(c, L, key);  // (ends with a barrier)
  const Scorer sc = c;
  stream_at_or_above(c, L.thr, [&](int id, uint32_t raw, int cc) {
    if (v3_bin_of_raw(raw) >= 0) take(key_of(sc.score_of(raw, cc)), id);  // (else a side element, taken above)
  });
  __syncthreads();
  const int n = min(*c.gbuf_n(), kCandCap);
  cand_sort(L, n);
  const float* noise_row = S.noise ? S.noise + (size_t)S.row * c.vocab : nullptr;
  const FinishOut r = finish_sorted(*c.x(), list, list + kCandCap, n, S.P, noise_row, &S.out);
  if (S.scores_out) {
    float* dst = S.scores_out + (size_t)S.row * c.vocab;
    for (int id = threadIdx.x; id < c.vocab; id += kThreads) dst[id] = __int_as_float(0xff800000);
    __syncthreads();
    for (int i = threadIdx.x; i < (int)r.n_kept; i += kThreads) dst[cand_id(list[i])] = score_of(cand_key(list[i]));
  }
  if (threadIdx.x == 0) {
    write_finish(r, &S.out);
    S.out.status |= S.status;
    if (S.tokens_out) S.tokens_out[S.row] = r.token;
    if ((S.flags & HS_SAMPLE_APPEND_TOKEN) && S.slot_ok && r.token >= 0 && r.token < c.vocab) {
      if (!slot_append_one(c.pool, S.P.slot, r.token)) S.out.status |= 2;
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) write_record(S.out_row, S.out, S.P.n_logprobs >= 0, S.mail_row, S.mail_tag);
  release_scratch(S);
  return true;
}

// From the row's count table (and rare tokens) to its record.
__device__ __forceinline__ void finish_counted_row() {
  CountState& S = count_state();
  Ctx3& c = S.c;
  const int tid = threadIdx.x;
  if (!phase_histogram()) {  // cannot happen while n_scratch covers the resident CTAs; fail the row, do not wait
    if (tid == 0) { S.out.token = 0; S.out.status = 128; S.out.n_top = 0; S.out.n_kept = 0; }
    __syncthreads();
    if (tid < 32) write_record(S.out_row, S.out, S.P.n_logprobs >= 0, S.mail_row, S.mail_tag);
    return;
  }
  if (is_candidate_row(S.P, c.vocab) && finish_listed_row()) return;
  if (c.greedy) {
    phase_greedy();
  } else {
    phase_cuts();
    phase_draw();
    __syncthreads();
    phase_mark(S, 14);
    int token = S.ask.token;
    if (S.ask.kind) token = phase_find();
    if (token < 0 || token == 0x7fffffff) {
      token = S.side_best ? (int)(~(uint32_t)(S.side_best & 0xffffffffu)) : 0;
      raise_status(S, 1);
    }
    put_state(S.token, token);
    __syncthreads();
  }
  phase_mark(S, 7);
  if (S.P.n_logprobs >= 0) phase_logprobs();
  // ---- optional dump of the final scores (parity tests)
  if (S.scores_out) {
    need_tie_limit();
    float* dst = S.scores_out + (size_t)S.row * c.vocab;
    const float ninf = __int_as_float(0xff800000);
#pragma unroll 1
    for (int id = tid; id < c.vocab; id += kThreads) {
      const float s = c.element_score(id, c.logits[id], c.class_of(id));
      dst[id] = (c.greedy || S.kept.has(key_of(s), id)) ? s : ninf;
    }
  }
  if (tid == 0) {
    const int token = S.token;
    S.out.token = token;
    S.out.n_kept = S.out.n_after_topp = (int32_t)S.n_kept;
    S.out.cut_bits = __float_as_uint(score_of(S.kept.cut_key));
    S.out.n_cut_ties = (int32_t)S.cut_ties;
    S.out.row_max = c.m;
    if (S.tokens_out) S.tokens_out[S.row] = token;
    // (a row for the general kernel is counted by that one)
    if ((S.flags & HS_SAMPLE_APPEND_TOKEN) && S.slot_ok && !(S.status & 4) && token >= 0 && token < c.vocab) {
      if (!slot_append_one(c.pool, S.P.slot, token)) S.status |= 2;
    }
    S.out.status = S.status;
  }
  __syncthreads();
  if (tid < 32) write_record(S.out_row, S.out, S.P.n_logprobs >= 0, S.mail_row, S.mail_tag);
  release_scratch(S);
  phase_mark(S, 9);
}

}  // namespace hs
