// The bf16 row kernel: one launch per step, one CTA per work item, two CTAs resident per SM.
// An item is a row for the counting path (hs_row_v3.cuh; also the plain arg-max rows of a
// mixed batch) or one part of a row for the candidate path (small top_k, hs_row_topk.cuh);
// the hardware hands the items out in grid order as SMs free up, the long ones first.  No CTA
// waits for another: the last part of a candidate row to arrive finishes that row, and a row
// whose candidate list overflowed is counted by the CTA that found out (and then listed after all).
#pragma once
#include <type_traits>

#include "hs_row_v3.cuh"
#include "hs_row_topk.cuh"
#include "hs_sharded.cuh"
#include "hs_row_finish.cuh"

namespace hs {

// One chunk of eight tokens the counting loop could not take in its branch-free form (a
// value outside the bin window, a token of count class 3): token by token, out of line so
// that the unrolled loop stays small.
__device__ __noinline__ void count_chunk_slow(uint32_t* tab, int* rare_n, int2* rare, uint4 w, uint32_t cl, int first) {
  const uint32_t words[4] = {w.x, w.y, w.z, w.w};
#pragma unroll 1
  for (int k = 0; k < 8; ++k) {
    const uint32_t raw = (words[k >> 1] >> (16 * (k & 1))) & 0xffffu;
    const int cc = (int)((cl >> (2 * k)) & 3u);
    if (cc == 3) continue;  // listed per request; scored individually with its exact count
    const int b = v3_bin_of_raw(raw);
    if (b >= 0) {
      atomicAdd(&tab[cc * kV3Bins + b], 1u);
    } else {
      const int slot = atomicAdd(rare_n, 1);
      if (slot < kV3RareCap) rare[slot] = make_int2(first + k, (int)(raw | ((uint32_t)cc << 16)));
    }
  }
}

// Counts the tokens of a row (also: plain arg max of a row in a mixed batch, start to end).  part < 0:
// this CTA counts the whole row.  part >= 0: the row's tokens are counted by args.csplit CTAs,
// each a contiguous range; every part leaves its counts and rare tokens in global scratch,
// and the part that arrives last (a ticket) adds the others' to its own.  True when this CTA has
// the whole row's counts and goes on.
__device__ __forceinline__ bool count_tokens(const RowV3Args& args, int row_index, int part) {
  const RowKernelArgs& a = args.base;
  CountState& S = count_state();
  const hs_row_params& P = S.P;
  hs_row_out* out = &S.out;
  const int tid = threadIdx.x;
  Ctx3 c;  // (this half's own copy, in registers)
  c.row = row_index;
  c.vocab = a.vocab;
  c.set_row(a.logits, a.row_stride);
  c.greedy = P.temperature == 0.0f;
  c.T = P.temperature;
  c.rp = P.repetition_penalty;
  c.pp = P.presence_penalty;
  c.fp = P.frequency_penalty;
  c.pool = a.pool;
  c.slot = P.slot;
  const bool slot_ok = P.slot >= 0 && P.slot < a.pool.slots_total;
  const bool penalised = slot_ok && (c.rp != 1.0f || c.pp != 0.0f || c.fp != 0.0f);
  c.cls = penalised ? a.pool.cls + (size_t)P.slot * a.pool.cls_stride : nullptr;
  c.s_pair = c.side();
  c.s_cap = kV3SideShared;
  c.n_s = 0;
  c.m = 0.f;
  if (tid == 0) {
    S.c = c;
    S.kept = KeptSet{0u, 0x7fffffff};
    S.q_kept = 0;
    S.n_kept = (u64)a.vocab;
    S.out.n_after_topk = S.out.n_after_minp = a.vocab;
    S.cut_group_cnt = 0;  // members at the cut key (kept or not)
    S.cut_ties = -1;
    S.status = P.slot >= a.pool.slots_total ? 64 : 0;  // a slot this sampler does not have: no penalties
    S.token = -1;
    S.scratch = -1;
    S.have_cut_group = S.tie_split = S.filled = false;
    S.slot_ok = slot_ok;
    S.penalised = penalised;
    S.row = row_index;
    S.flags = (int)a.flags;
    S.token_draw = a.token_draw;
    S.s_cap_all = args.s_cap;
    S.n_scratch = args.n_scratch;
    S.s_pair_all = args.s_pair;
    S.scratch_busy = args.scratch_busy;
    S.noise = a.noise;
    S.scores_out = a.scores_out;
    S.tokens_out = a.tokens_out;
    S.out_row = record_of(a, row_index);
    S.mail_row = mail_of(a, row_index);
    S.mail_tag = a.mail_tag;
    S.parts = part < 0 ? 1 : args.csplit;
    S.lists = args.ctab + (size_t)row_index * args.csplit * kHandedCap;
    S.lens = args.crare_n + (size_t)row_index * args.csplit;
    S.clocks = args.phase_clocks ? args.phase_clocks + (size_t)row_index * kV3PhaseSlots : nullptr;
    if (S.clocks) S.clocks[0] = clock64();
  }
  int2* rare = c.rare();
  uint32_t* staged = at_smem<kLayV3.staged, uint32_t>();
  int* small = count_small();
  int* rare_n = small + 1;
  int* defer_n = small + 27;
  int* defer = at_smem<kLayV3.defer, int>();

  // ---- plain greedy rows of a mixed batch: arg max only -----------------------------------
  if (c.greedy && !penalised && P.n_logprobs < 0) {
    if (part > 0) return false;  // (one CTA walks the whole row)
    u64 best = 0;
    auto consider = [&](uint32_t raw, int id) {
      const u64 packed = ((u64)key_of(canonical(__uint_as_float(raw << 16))) << 32) | (uint32_t)(~(uint32_t)id);
      best = packed > best ? packed : best;
    };
    for (int i = tid; i < c.n8(); i += kThreads) {
      const uint4 w = __ldcg(c.chunks() + i);
      const uint32_t words[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int k = 0; k < 8; ++k) consider((words[k >> 1] >> (16 * (k & 1))) & 0xffffu, c.first_of(i) + k);
    }
    if (tid < c.n_loose()) consider(c.logits[c.loose(tid)], c.loose(tid));
    best = block_max_u64(*c.x(), best);
    if (a.scores_out) {
      float* dst = a.scores_out + (size_t)c.row * a.vocab;
      for (int id = tid; id < c.vocab; id += kThreads) dst[id] = canonical(__uint_as_float((uint32_t)c.logits[id] << 16));
    }
    if (tid == 0) {
      out->token = (int)(~(uint32_t)(best & 0xffffffffu));
      if (a.tokens_out) a.tokens_out[c.row] = out->token;
      out->logprob = 0.f; out->n_top = 0; out->status = S.status;
      out->n_kept = a.vocab; out->n_after_topk = a.vocab; out->n_after_minp = a.vocab; out->n_after_topp = a.vocab;
      out->cut_bits = 0xff800000u; out->n_cut_ties = -1;
      out->row_max = score_of((uint32_t)(best >> 32)); out->log_z = 0.f;
    }
    __syncthreads();
    if (tid < 32) write_record(record_of(a, c.row), *out, false, mail_of(a, c.row), a.mail_tag);
    return false;
  }

  // this CTA's range of 8-token chunks [chunk_lo, chunk_hi); the last part also takes the row's
  // loose tokens
  const int n8_row = c.n8();
  const int parts = part < 0 ? 1 : args.csplit;
  const int my_part = part < 0 ? 0 : part;
  const int per_part = chunks_per_part(n8_row, parts);
  const int chunk_lo = min(my_part * per_part, n8_row), chunk_hi = min(chunk_lo + per_part, n8_row);
  const bool last_part = my_part == parts - 1;
  // small[16..18] / [19..21]: highest (+ 1) / lowest non-empty cell per count class; [22]: lowest side key
  if (tid < 64) small[tid] = (tid >= 19 && tid <= 22) ? -1 : 0;
  if (tid == 0) c.x()->bcast[5] = 0;  // highest side element, (key, ~id)
  __syncthreads();
  for (int i = tid; i < kCells / 4; i += kThreads) reinterpret_cast<uint4*>(c.tab())[i] = make_uint4(0u, 0u, 0u, 0u);
  cudaGridDependencySynchronize();  // (the histograms are up to date from here on)
  __syncthreads();
  // ---- A. the one read of the row from HBM: count tokens per (count class, value) --------
  {
    auto count_one = [&](uint32_t raw, int cc, int id) {
      if (cc == 3) return;  // listed per request; handled below with its exact count
      const int b = v3_bin_of_raw(raw);
      if (b >= 0) {
        atomicAdd(&c.tab()[cc * kV3Bins + b], 1u);
      } else {
        const int slot = atomicAdd(rare_n, 1);
        if (slot < kV3RareCap) rare[slot] = make_int2(id, (int)(raw | ((uint32_t)cc << 16)));
      }
    };
    const uint4* src4 = c.chunks();
    const bool has_cls = c.cls != nullptr;
    // Eight tokens at a time without a branch per token.  Per 32-bit word (two tokens):
    // |x| + (0x8000 - base) sets bit 15 of a half iff |x| >= base and leaves |x| - base in its
    // low bits; |x| + (0x8000 - top) sets it iff |x| >= top; a byte permute with sign
    // replication turns the two sign bits into two 16-bit masks, and one LOP3 leaves, per half,
    // the bin relative to the middle of a class table as a signed 16-bit number (idx for
    // x >= 0, -1 - idx for x < 0).  Per token: sign-extending extraction (one permute), class
    // offset and table address (two multiply-adds on the FMA pipe), the reduction.  A chunk
    // with a value outside the window or a token of count class 3 (rare) takes the per-token
    // path.  Written as PTX where one instruction is meant.
    constexpr uint32_t kLoAdd = (0x8000u - kV3Base) * 0x00010001u;
    constexpr uint32_t kHiAdd = (0x8000u - (kV3Base + (uint32_t)kV3Half)) * 0x00010001u;
    constexpr uint32_t kClassBytes = (uint32_t)(kV3Bins * 4);
    const uint32_t tab_mid = (uint32_t)__cvta_generic_to_shared(c.tab() + kV3Half);
    auto take_chunk = [&](const uint4& w4, uint32_t cl4, int i) {
      const uint32_t words[4] = {w4.x, w4.y, w4.z, w4.w};
      uint32_t rel2[4];
      uint32_t wnd = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint32_t mag, mask;
        asm("and.b32 %0, %1, 0x7fff7fff;" : "=r"(mag) : "r"(words[k]));
        const uint32_t lo = mag + kLoAdd, ht = mag + kHiAdd;
        asm("lop3.b32 %0, %1, %2, %3, 0xef;" : "=r"(wnd) : "r"(lo), "r"(ht), "r"(wnd));     // wnd | ~lo | ht
        asm("prmt.b32 %0, %1, 0, 0xBB99;" : "=r"(mask) : "r"(words[k]));                     // 0xffff per negative half
        asm("lop3.b32 %0, %1, 0x7fff7fff, %2, 0x6a;" : "=r"(rel2[k]) : "r"(lo), "r"(mask));  // (lo & 0x7fff7fff) ^ mask
      }
      // bits 15 / 31 of wnd: a value outside the window; bit 2J of cl & (cl >> 1): token J is of class 3
      if (((wnd & 0x80008000u) | (cl4 & (cl4 >> 1) & 0x5555u)) == 0) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int kShift = 2 * (2 * k + h);
            uint32_t r;
            if (h == 0) asm("prmt.b32 %0, %1, 0, 0x9910;" : "=r"(r) : "r"(rel2[k]));  // low half, sign extended
            else asm("prmt.b32 %0, %1, 0, 0xBB32;" : "=r"(r) : "r"(rel2[k]));          // high half, sign extended
            uint32_t base;
            if (kShift < 14) base = (cl4 & (3u << kShift)) * (kClassBytes >> kShift) + tab_mid;
            else base = (cl4 >> 14) * kClassBytes + tab_mid;
            const uint32_t addr = r * 4u + base;
            asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(addr) : "memory");
          }
        }
      } else {
        // set aside: a call here would save and restore the loop's registers through local
        // memory (round trips to L2 with this kernel's small L1), a few thousand cycles a time
        const int slot = atomicAdd(defer_n, 1);
        if (slot < kV3DeferCap) defer[slot] = i;
      }
    };
    // Two batches of loads: the next one is on its way while this one is counted.  The main
    // loop runs without bounds checks; what is left over is taken chunk by chunk.
    constexpr int kInFlight = 2;  // 128-bit loads per thread and batch
    constexpr int kStride = kInFlight * kThreads;
    // (one copy of the loop per way to get at the count classes: the question is not asked per chunk)
    auto count_chunks = [&](auto classes) {
      const int n_full = (chunk_hi - chunk_lo) / kStride;
      int i0 = chunk_lo + tid;
      if (n_full > 0) {
        uint4 w[kInFlight], wn[kInFlight];
        uint32_t cl[kInFlight], cn[kInFlight];
#pragma unroll
        for (int u = 0; u < kInFlight; ++u) {
          w[u] = __ldcg(src4 + i0 + u * kThreads);  // past L1: almost all of it is shared memory here
          cl[u] = classes(i0 + u * kThreads);
          wn[u] = w[u];
          cn[u] = cl[u];
        }
        for (int it = 0; it < n_full; ++it) {
          if (it + 1 < n_full) {
#pragma unroll
            for (int u = 0; u < kInFlight; ++u) {
              wn[u] = __ldcg(src4 + i0 + kStride + u * kThreads);
              cn[u] = classes(i0 + kStride + u * kThreads);
            }
          }
#pragma unroll
          for (int u = 0; u < kInFlight; ++u) take_chunk(w[u], cl[u], i0 + u * kThreads);
#pragma unroll
          for (int u = 0; u < kInFlight; ++u) { w[u] = wn[u]; cl[u] = cn[u]; }
          i0 += kStride;
        }
      }
      for (int i = i0; i < chunk_hi; i += kThreads) take_chunk(__ldcg(src4 + i), classes(i), i);
    };
    if (!has_cls) {
      count_chunks([](int) { return 0u; });
    } else if (c.head() == 0) {
      const unsigned short* cls16 = reinterpret_cast<const unsigned short*>(c.cls);
      count_chunks([cls16](int i) { return (uint32_t)__ldcg(cls16 + i); });
    } else {
      count_chunks([&c](int i) { return c.chunk_classes(i); });
    }
    // the chunks that were set aside, token by token, one thread per chunk
    __syncthreads();
    {
      const int n_defer = *defer_n;
      if (n_defer <= kV3DeferCap) {
        for (int j = tid; j < n_defer; j += kThreads) {
          const int i = defer[j];
          count_chunk_slow(c.tab(), rare_n, rare, __ldcg(src4 + i), has_cls ? c.chunk_classes(i) : 0u, c.first_of(i));
        }
      } else {
        // more than the list holds (a row full of values outside the bin window): every chunk of
        // the range is looked at again and those the loop did not take are counted now
        for (int i = chunk_lo + tid; i < chunk_hi; i += kThreads) {
          const uint4 w4 = __ldcg(src4 + i);
          const uint32_t cl4 = has_cls ? c.chunk_classes(i) : 0u;
          const uint32_t words[4] = {w4.x, w4.y, w4.z, w4.w};
          bool slow = (cl4 & (cl4 >> 1) & 0x5555u) != 0u;
#pragma unroll
          for (int q = 0; q < 8; ++q) slow = slow || v3_bin_of_raw((words[q >> 1] >> (16 * (q & 1))) & 0xffffu) < 0;
          if (slow) count_chunk_slow(c.tab(), rare_n, rare, w4, cl4, c.first_of(i));
        }
      }
    }
    if (last_part && tid < c.n_loose()) count_one(c.logits[c.loose(tid)], c.class_of(c.loose(tid)), c.loose(tid));
  }
  __syncthreads();
  if (parts > 1) {
    // Hand this part's counts over, as a list of (class, count), with its rare tokens; then a ticket.
    // The part that draws the last ticket adds the other parts' lists to its own table and goes on;
    // the others are done.  Nobody waits for anybody.  (Lists instead of whole tables: about 16 KB a
    // part instead of 72.)  Bound by the banks when a list is added up, and by the round trips to L2: in the
    // order of the cells, four entries a load and the next piece under way (by thread, one entry a load and list
    // by list, and without the look-up in nth_in_parts, a call of one row of 248,320 took 107.6 us and 97.2 this way, when
    // such a row was cut in sixteen; with the seven parts of now it takes 87.4).
    const size_t mine = (size_t)c.row * parts + my_part;
    const int nr = *rare_n;
    for (int t = tid; t < min(nr, kV3RareCap); t += kThreads) args.crare[mine * kV3RareCap + t] = rare[t];
    {
      // Warp w lists the w-th run of cells, 32 neighbours at a time, so that a list is in the order of
      // the cells: whoever adds it up finds neighbouring entries in different banks, and can look a
      // class up in it (nth_in_parts).  A count that 17 bits do not hold takes several entries, side by side.
      const int lane = tid & 31, warp = tid >> 5;
      const int rows = (c.cls ? kCells : kV3Bins) / (32 * kWarps);  // (without penalties there is one count class)
      static_assert(kV3Bins % (32 * kWarps) == 0, "every warp has whole groups of 32 cells");
      const int first = warp * rows * 32 + lane;
      const uint32_t* run = c.tab() + first;
      int n = 0;
#pragma unroll 4
      for (int u = 0; u < rows; ++u) {
        const uint32_t v = run[32 * u];
        n += v ? 1 : 0;
        if (v > kMostHanded) n += (int)((v - 1u) / kMostHanded);
      }
      n = __reduce_add_sync(0xffffffffu, n);
      if (lane == 0) small[48 + warp] = n;
      __syncthreads();  // (the rare tokens have left, too)
      const int of_warp = lane < kWarps ? small[48 + lane] : 0;
      const int total = __reduce_add_sync(0xffffffffu, of_warp);
      int at = __reduce_add_sync(0xffffffffu, lane < warp ? of_warp : 0);
      uint32_t* gtab = args.ctab + mine * kHandedCap;
      uint32_t* dst = total <= kV3Staged ? staged : gtab;
#pragma unroll 1
      for (int u = 0; u < rows; ++u) {
        uint32_t v = run[32 * u];
        const uint32_t cell = (uint32_t)(first + 32 * u);
        const uint32_t who = __ballot_sync(0xffffffffu, v != 0u);
        if (!__any_sync(0xffffffffu, v > kMostHanded)) {
          if (v) dst[at + __popc(who & ((1u << lane) - 1u))] = cell | (v << 15);
          at += __popc(who);
        } else {
          const int entries = v ? 1 + (int)((v - 1u) / kMostHanded) : 0;
          int incl = entries;
#pragma unroll 1
          for (int d = 1; d < 32; d <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += o;
          }
#pragma unroll 1
          for (int to = at + incl - entries; v; ++to) {
            const uint32_t part_v = min(v, kMostHanded);
            dst[to] = cell | (part_v << 15);
            v -= part_v;
          }
          at += __shfl_sync(0xffffffffu, incl, 31);
        }
      }
      __syncthreads();
      if (dst == staged)
        for (int i = tid; i < (total + 3) / 4; i += kThreads)
          reinterpret_cast<uint4*>(gtab)[i] = reinterpret_cast<const uint4*>(staged)[i];
      if (tid == 0) args.crare_n[mine] = make_int2(total, nr);
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) small[14] = atomicAdd(&args.count_ticket[c.row], 1);
    __syncthreads();
    if (small[14] != parts - 1) return false;
    __threadfence();
    if (tid == 0) args.count_ticket[c.row] = 0;
    // The other parts' lists, piece by piece of up to 4,096 entries, the next piece's on their way while this
    // one's are added.
    const int2* lens = args.crare_n + (size_t)c.row * parts;
    const uint32_t* lists = args.ctab + (size_t)c.row * parts * kHandedCap;
    int2* part_len = reinterpret_cast<int2*>(defer);  // (the staged list has left)
    if (tid < parts) part_len[tid] = __ldcg(lens + tid);
    __syncthreads();
    constexpr int kFlight = 2;  // four entries each
    struct Piece { int g, at; } next{my_part == 0 ? 1 : 0, 0};
    auto fetch = [&](uint4 (&v)[kFlight]) {
      if (next.g >= parts) return;
      const int n = part_len[next.g].x, n4 = (n + 3) >> 2;
      const uint4* src = reinterpret_cast<const uint4*>(lists + (size_t)next.g * kHandedCap);
#pragma unroll
      for (int u = 0; u < kFlight; ++u) {
        const int i = next.at + tid + u * kThreads;
        v[u] = i < n4 ? __ldcg(src + i) : make_uint4(0u, 0u, 0u, 0u);
        if (i == n4 - 1) {  // (nothing is behind a list's last entry)
          if (4 * i + 1 >= n) v[u].y = 0u;
          if (4 * i + 2 >= n) v[u].z = 0u;
          if (4 * i + 3 >= n) v[u].w = 0u;
        }
      }
      next.at += kFlight * kThreads;
      if (next.at >= n4) {
        next.at = 0;
        next.g += next.g + 1 == my_part ? 2 : 1;
      }
    };
    uint4 v[kFlight], vn[kFlight];
    fetch(v);
    for (bool more = true; more;) {
      more = next.g < parts;
      fetch(vn);
#pragma unroll
      for (int u = 0; u < kFlight; ++u) {
        const uint32_t e[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (e[k]) atomicAdd(&c.tab()[e[k] & 0x7fffu], e[k] >> 15);
        v[u] = vn[u];
      }
    }
    int n_rare_all = 0;
#pragma unroll 1
    for (int g = 0; g < parts; ++g) {
      // (a total beyond the capacity is swept up below)
      const int n = part_len[g].y;
      for (int t = tid; t < min(n, kV3RareCap); t += kThreads)
        if (n_rare_all + t < kV3RareCap) rare[n_rare_all + t] = __ldcg(args.crare + ((size_t)c.row * parts + g) * kV3RareCap + t);
      n_rare_all += n;
    }
    if (tid == 0) *rare_n = n_rare_all;
    __syncthreads();
  }
  phase_mark(S, 1);
  return true;
}

// One part of a candidate row (a contiguous range of its tokens).  The CTA that brings in the
// row's last part finishes the row.  Returns true when the row's candidate list overflowed
// and the caller (the finishing CTA) has to count the row after all.
__device__ __forceinline__ bool cand_part(const RowV3Args& args, unsigned char* smem_raw, const hs_row_params& P,
                                          hs_row_out* out, int row_index, int part) {
  const RowKernelArgs& a = args.base;
  const LayoutCand lay = layout_cand();
  Ctx3 c;
  int* small = reinterpret_cast<int*>(smem_raw + lay.small);
  CandCtx L{reinterpret_cast<u64*>(smem_raw + lay.cand), small + 4, small + 5,
            reinterpret_cast<uint32_t*>(smem_raw + lay.count), small + 8, nullptr};
  const int tid = threadIdx.x;
  c.row = row_index;
  c.vocab = a.vocab;
  c.greedy = false;
  // the row is streamed by args.split CTAs, each taking a contiguous range of tokens
  const int split = args.split;
  c.set_row(a.logits, a.row_stride);
  const int width = (c.n8() + split - 1) / split;
  c.chunk_lo = min(part * width, c.n8());
  c.chunk_hi = min(c.chunk_lo + width, c.n8());
  c.lo = part == 0 ? 0 : c.first_of(c.chunk_lo);
  c.hi = part == split - 1 ? a.vocab : c.first_of(c.chunk_hi);
  c.T = P.temperature; c.rp = P.repetition_penalty; c.pp = P.presence_penalty; c.fp = P.frequency_penalty;
  c.pool = a.pool;
  c.slot = P.slot;
  const bool slot_ok = P.slot >= 0 && P.slot < a.pool.slots_total;
  const bool penalised = slot_ok && (c.rp != 1.0f || c.pp != 0.0f || c.fp != 0.0f);
  c.cls = penalised ? a.pool.cls + (size_t)P.slot * a.pool.cls_stride : nullptr;
  c.s_pair = nullptr; c.n_s = 0; c.s_cap = 0; c.m = 0.f;
  unsigned long long* clocks = args.phase_clocks ? args.phase_clocks + (size_t)c.row * kV3PhaseSlots : nullptr;
  auto mark = [&](int slot) {
    if (clocks && tid == 0) clocks[slot] = clock64();
  };
  mark(0);
  L.dbg = clocks;
  if (tid < 16) small[tid] = 0;
  __syncthreads();
  int n = c.hi > c.lo ? topk_candidates(c, L, min(P.top_k, c.hi - c.lo)) : 0;
  mark(1);
  u64* mass = reinterpret_cast<u64*>(smem_raw + lay.mass);
  // a lone CTA cuts its list at the k-th highest score now, and sorts it; a part of a split row hands
  // its candidates over as they are unless they would crowd the merged list
  if (n > 0) {
    const bool cut = n > P.top_k && (split == 1 || n > kCandCap / split);
    const uint32_t bound = cut ? cand_kth_key(*c.x(), L, n, P.top_k) : 0u;
    mark(14);
    // (without a cut the pass still drops the entries the scoring voided)
    n = split == 1 ? cand_keep_sorted(L, mass, n, bound) : cand_compact(L, n, bound);
  }
  if (split > 1) {
    // hand this CTA's candidates over; the CTA that arrives last finishes the row
    static_assert(kSplitCap >= kCandCap, "a part's whole list fits in its hand-over block");
    u64* mine = args.split_lists + ((size_t)c.row * split + part) * kSplitCap;
    for (int i = tid; i < n; i += kThreads) mine[i] = L.cand[i];
    if (tid == 0) args.split_n[c.row * split + part] = n;  // -1: this part overflowed
    __threadfence();
    __syncthreads();
    if (tid == 0) small[6] = atomicAdd(&args.split_ticket[c.row], 1);
    __syncthreads();
    if (small[6] != split - 1) return false;
    mark(12);
    __threadfence();
    if (tid == 0) args.split_ticket[c.row] = 0;
    // all parts' lengths first, then all copies at once (one wait instead of one per part)
    if (tid < split) small[12 + tid] = ((volatile int*)args.split_n)[c.row * split + tid];  // -1: that part overflowed
    __syncthreads();
    {
      int at = 0;
      bool overflow = false;
      for (int g = 0; g < split; ++g) {
        const int ng = small[12 + g];
        if (ng < 0) { overflow = true; continue; }
        const u64* theirs = args.split_lists + ((size_t)c.row * split + g) * kSplitCap;
        for (int i = tid; i < ng; i += kThreads)
          if (at + i < kCandCap) L.cand[at + i] = ((volatile const u64*)theirs)[i];
        at += ng;
      }
      n = (overflow || at > kCandCap) ? -1 : at;
    }
    __syncthreads();
    mark(13);
    if (n >= 0) {
      const uint32_t bound = n > kSortAll ? cand_kth_key(*c.x(), L, n, P.top_k) : 0u;
      mark(14);
      n = cand_keep_sorted(L, mass, n, bound);
    }
  }
  if (n < 0) return true;  // more than a candidate list holds: the row is counted
  mark(15);
  if (n > P.top_k) {
    // a list that was sorted whole: top-k keeps the first k entries and the ties of the k-th
    const uint32_t cut = cand_key(L.cand[P.top_k - 1]);
    u64 keep = 0, unused = 0;
    for (int i = tid; i < n; i += kThreads) keep += cand_key(L.cand[i]) >= cut ? 1 : 0;
    block_sum2(*c.x(), keep, unused);
    n = (int)keep;
  }
  mark(2);
  const float* noise_row = a.noise ? a.noise + (size_t)c.row * a.vocab : nullptr;
  FinishOut r = finish_sorted(*c.x(), L.cand, mass, n, P, noise_row, out, clocks);
  if (P.slot >= a.pool.slots_total) r.status |= 64;  // a slot this sampler does not have: no penalties
  if (a.scores_out) {
    float* dst = a.scores_out + (size_t)c.row * a.vocab;
    for (int id = tid; id < c.vocab; id += kThreads) dst[id] = __int_as_float(0xff800000);
    __syncthreads();
    for (int i = tid; i < (int)r.n_kept; i += kThreads) dst[cand_id(L.cand[i])] = score_of(cand_key(L.cand[i]));
  }
  if (tid == 0) {
    write_finish(r, out);
    if (a.tokens_out) a.tokens_out[c.row] = r.token;
    if ((a.flags & HS_SAMPLE_APPEND_TOKEN) && slot_ok && r.token >= 0 && r.token < a.vocab) {
      if (!slot_append_one(a.pool, P.slot, r.token)) out->status = r.status | 2;
    }
  }
  __syncthreads();
  if (tid < 32) write_record(record_of(a, c.row), *out, P.n_logprobs >= 0, mail_of(a, c.row), a.mail_tag);
  mark(8);
  return false;
}

// Shared memory of the persistent kernel: the larger of the two paths' layouts.
__host__ __device__ inline size_t bf16_kernel_smem() {
  const size_t a = layout_v3().total, b = layout_cand().total;
  return a > b ? a : b;
}

// One CTA per work item, two CTAs resident per SM; the hardware hands out the items in grid
// order, long ones first: batch * csplit items = part p of row r on the counting path (a CTA
// whose row is not a counting row leaves at once), then batch * split items = part p of row r
// on the candidate path (likewise).  No CTA waits for another.
__global__ void __launch_bounds__(kThreads, 2) row_kernel_bf16(const __grid_constant__ RowV3Args args,
                                                               const __grid_constant__ InlineRows inl) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  CountState& S = count_state();
  hs_row_params& P = S.P;  // (shared: in registers its twelve words would be spilled)
  hs_row_out& record = S.out;
  const int item = blockIdx.x;
  const int n_count = args.batch * args.csplit;
  bool count = item < n_count;
  // counting items are laid out part-major, so that the parts of one row start on different SMs
  int row = count ? item % args.batch : (item - n_count) / args.split;
  int part = count ? item / args.batch : (item - n_count) % args.split;
  if (threadIdx.x == 0) P = row_params(args.base, inl, row);
  __syncthreads();
  if (is_candidate_row(P, args.base.vocab) == count) return;  // the other path's row
  if (threadIdx.x < sizeof(hs_row_out) / 4) reinterpret_cast<uint32_t*>(&record)[threadIdx.x] = 0u;
  __syncthreads();
  // (tuning aid: when each item started and ended, in ns of the global timer, slots 48.. of its row)
  unsigned long long* when = nullptr;
  if (args.phase_clocks && threadIdx.x == 0 && part < 4) {
    when = args.phase_clocks + (size_t)row * kV3PhaseSlots + (count ? 48 : 56) + 2 * part;
    when[0] = global_timer_ns();
  }
  if (!count) {
    if (!cand_part(args, smem_raw, P, &record, row, part)) {
      if (when) when[1] = global_timer_ns();
      return;
    }
    __syncthreads();
    part = -1;  // more than a candidate list holds: this CTA counts the whole row
  } else if (args.csplit == 1) {
    part = -1;
  }
  if (count_tokens(args, row, part)) finish_counted_row();
  if (when) when[1] = global_timer_ns();
}

}  // namespace hs
