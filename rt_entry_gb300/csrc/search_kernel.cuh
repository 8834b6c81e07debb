// search_kernel.cuh -- persistent warp-per-query beam search for sm_103a.
//
// Computes exactly what the reference's GraphSearchKernel computes
// (graph_search.cuh:56-1964, one 64-thread block per query), reorganised for
// one warp per query:
//   * the pool (L = 32*NL slots, or 16 slots for NL = 0) and the batch
//     (B = 32*NB slots) live in registers: slot p sits in lane p%32,
//     register p/32.  The few candidates of a batch are compacted in shared
//     memory and inserted or placed by rank, which gives the reference's
//     result whenever they are distinct and the pool is sorted; ties, larger
//     counts, and all batches of a query from its first NaN on run its
//     comparator network (bitonic batch sort, pool/batch merge,
//     half-cleaner, graph_search.cuh:888-957 and :1424-1493) on those
//     registers, across lanes through shuffles and inside a lane for
//     distances >= 32;
//   * base rows are stored lane-interleaved (see layout.cuh): one 128-bit
//     load gives lane l the dims l, l+32, l+64, l+96 -- exactly the dims the
//     reference's reduction tree assigns to lane l -- so a neighbour row is a
//     single fully coalesced 512-byte gather at d = 128;
//   * distances of up to 16 neighbours are reduced together by a butterfly
//     whose every addition pairs the same partial sums as the reference's
//     shuffle-down tree (16,8,4,2,1), so the results are bit-identical while
//     using one shuffle per neighbour instead of five;
//   * the visited-set bloom filter lives in shared memory per warp, sized at
//     run time (the reference fixes 512 words, graph_search.cuh:4-5);
//   * warps pull queries from an atomic counter until none are left; a
//     batch larger than the resident warps is pulled through a permutation
//     that groups its queries by entry leaf (SearchArgs::order), so that
//     the queries running at the same time share rows in L2.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <stdint.h>

#include <type_traits>

#include "layout.cuh"
#include "pdl.cuh"
#include "search_types.h"

namespace rte {

constexpr float kMaxDist = 536870912.0f;  // (float)0x1fffffff, structure_on_device.cuh:6
constexpr unsigned kFull = 0xffffffffu;

// Bloom-filter hash multipliers (graph_search.cuh:89-97).
__constant__ uint32_t c_hash_mul[20] = {
    0x924ed183U, 0xd854fc0aU, 0xecf5e3b7U, 0x1bead407U, 0x28a30449U,
    0xbfc4d99fU, 0x715030e2U, 0xffcfb45bU, 0x6e4ce166U, 0xeb53c362U,
    0xa93c4f40U, 0xcecde0a4U, 0x0288592dU, 0x362c37bcU, 0x9d4824f0U,
    0xfdbdd68bU, 0x63258c85U, 0x6726905cU, 0x609500f9U, 0x4de48422U};


__device__ __forceinline__ uint32_t bloom_hash(int h, uint32_t x, uint32_t mask_bits) {
  // hash_ (graph_search.cuh:13-22); x % (SIZE<<5) with SIZE a power of two.
  x ^= x >> 16;
  x *= c_hash_mul[h << 1];
  x ^= x >> 13;
  x *= c_hash_mul[(h << 1) + 1];
  x ^= x >> 16;
  return x & mask_bits;
}

struct Bloom {
  uint32_t* w;
  uint32_t sw;          // w as a shared-space address
  uint32_t words_mask;  // words - 1
  uint32_t bits_mask;   // 32*words - 1
  int lw;               // log2(words)
  int nh;
  // set_bit / test_bit: word x % SIZE, bit x / SIZE (graph_search.cuh:7-28).
  // The first kUnrolled hashes have no branch between them: a test computes
  // all of them and issues its loads together, an id's hashes are computed
  // once for its test and its add, and an id that is not to be added (or a
  // hash beyond nh) ORs a zero instead of branching around the OR.  Measured
  // on one GB300 with one warp on an SM, testing, adding and compacting 64
  // ids: 1163 cycles with a branch per hash and around each add, 412 with
  // predicated ORs, 254 this way.  Further hashes (up to 10) run in a loop.
  static constexpr int kUnrolled = 3;
  __device__ __forceinline__ void set(uint32_t b, uint32_t on) const {
    asm volatile("red.shared.or.b32 [%0], %1;" ::"r"(sw + 4 * (b & words_mask)), "r"(on << (b >> lw)) : "memory");
  }
  __device__ __forceinline__ uint32_t word(uint32_t b) const {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(sw + 4 * (b & words_mask)) : "memory");
    return v;
  }
  __device__ __forceinline__ void hash(uint32_t x, uint32_t (&b)[kUnrolled]) const {
#pragma unroll
    for (int h = 0; h < kUnrolled; ++h) b[h] = bloom_hash(h, x, bits_mask);
  }
  // Adds x where on = 1 (0: nothing is added); the warp's lanes all call it.
  __device__ __forceinline__ void add(uint32_t (&b)[kUnrolled], uint32_t on) const {
#pragma unroll
    for (int h = 0; h < kUnrolled; ++h) set(b[h], h < nh ? on : 0u);
  }
  // The hashes from kUnrolled on, if there are any.
  __device__ __forceinline__ void add_more(uint32_t x, uint32_t on) const {
#pragma unroll 1
    for (int h = kUnrolled; h < nh; ++h) set(bloom_hash(h, x, bits_mask), on);
  }
  __device__ __forceinline__ void add(uint32_t x, uint32_t on) const {
    uint32_t b[kUnrolled];
    hash(x, b);
    add(b, on);
    add_more(x, on);
  }
  __device__ __forceinline__ bool test(const uint32_t (&b)[kUnrolled]) const {
    uint32_t v[kUnrolled];
#pragma unroll
    for (int h = 0; h < kUnrolled; ++h) v[h] = word(b[h]);
    uint32_t ok = 1u;
#pragma unroll
    for (int h = 0; h < kUnrolled; ++h) ok &= (v[h] >> (b[h] >> lw)) | (h < nh ? 0u : 1u);
    return ok != 0u;
  }
  __device__ __forceinline__ bool test_more(uint32_t x) const {
    bool ok = true;
#pragma unroll 1
    for (int h = kUnrolled; h < nh; ++h) {
      const uint32_t c = bloom_hash(h, x, bits_mask);
      ok &= ((word(c) >> (c >> lw)) & 1u) != 0u;
    }
    return ok;
  }
  __device__ __forceinline__ bool test(uint32_t x) const {
    uint32_t b[kUnrolled];
    hash(x, b);
    return test(b) & test_more(x);
  }
  // The filter starts on a 16-byte boundary and holds at least 32 words.
  __device__ __forceinline__ void clear(int lane) const {
    uint4* w4 = reinterpret_cast<uint4*>(w);
    for (uint32_t i = lane; i <= (words_mask >> 2); i += 32) w4[i] = make_uint4(0u, 0u, 0u, 0u);
  }
};

template <int V>
using Const = std::integral_constant<int, V>;

template <int N>
__device__ __forceinline__ int pick(const int (&a)[N], int c) {
  int v = a[0];
#pragma unroll
  for (int j = 1; j < N; ++j)
    if (c == j) v = a[j];
  return v;
}

// Compare-exchange of slot p with slot p^sub held by another lane (sub < 32).
// `desc` is the direction of the pair; both lanes evaluate the same
// predicate on (lower, upper), so ties never swap (strict comparisons).
__device__ __forceinline__ void cx_lanes(float& d, int& id, int sub, bool desc, int lane) {
  float od = __shfl_xor_sync(kFull, d, sub);
  int oi = __shfl_xor_sync(kFull, id, sub);
  bool lower = (lane & sub) == 0;
  float da = lower ? d : od;
  float db = lower ? od : d;
  bool sw = desc ? (da < db) : (da > db);
  if (sw) {
    d = od;
    id = oi;
  }
}

__device__ __forceinline__ void cx_regs(float& da, int& ia, float& db, int& ib, bool desc) {
  bool sw = desc ? (da < db) : (da > db);
  if (sw) {
    float t = da;
    da = db;
    db = t;
    int u = ia;
    ia = ib;
    ib = u;
  }
}

// Pool geometry: NL registers of 32 slots each, or NL == 0 for a 16-slot pool
// (beam 16) held in lanes 0..15 of one register; lanes 16..31 of that
// register keep (MAX, np) padding that no step ever reads back.
__host__ __device__ constexpr int pool_slots(int NL) { return NL == 0 ? 16 : 32 * NL; }
__host__ __device__ constexpr int pool_regs(int NL) { return NL == 0 ? 1 : NL; }
// Batch geometry: NB registers of 32 slots, or NB == 0 for a 16-slot batch
// (search width 1 over a degree-16 graph) in lanes 0..15 of one register;
// lanes 16..31 then hold (MAX, np) padding.
__host__ __device__ constexpr int batch_slots(int NB) { return NB == 0 ? 16 : 32 * NB; }
__host__ __device__ constexpr int batch_regs(int NB) { return NB == 0 ? 1 : NB; }
// Query registers per lane: C, or one unused register for the kernels built
// for any chunk count (C == 0), which keep the query in shared memory.
__host__ __device__ constexpr int qregs(int C) { return C == 0 ? 1 : C; }

// Bitonic sort of N slots (graph_search.cuh:888-919), N = 32*NB by default or
// 16 for the one-register beam-16 pool.  With DESC_FINAL the pair (a, a+sub)
// is descending when a's 2*step block index is even, so the result is
// descending, as the reference sorts its batch; otherwise the directions are
// mirrored and the result is ascending.  The stages are loops, not unrolled
// code: the network runs only where equal distances or many candidates ask
// for it (rank_candidates), and unrolled (36 stages x 8 registers for 256
// slots) it made the kernels larger than the instruction cache, which on
// one GB300 cost the 256-slot kernels 10 stalled cycles per issued
// instruction.
template <int NB, bool DESC_FINAL = true, int N = 32 * NB>
__device__ __forceinline__ void sort_batch_desc(float (&d)[NB], int (&id)[NB], int lane) {
  constexpr int B = N;
#pragma unroll 1
  for (int step = 1; step <= B / 2; step <<= 1) {
#pragma unroll
    for (int rs = NB / 2; rs >= 1; rs >>= 1) {
      if (rs > (step >> 5)) continue;
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        if (j & rs) continue;
        cx_regs(d[j], id[j], d[j + rs], id[j + rs], (((j << 5) & (2 * step)) == 0) == DESC_FINAL);
      }
    }
#pragma unroll 1
    for (int sub = step < 16 ? step : 16; sub >= 1; sub >>= 1) {
#pragma unroll
      for (int j = 0; j < NB; ++j)
        cx_lanes(d[j], id[j], sub, ((((j << 5) + lane) & (2 * step)) == 0) == DESC_FINAL, lane);
    }
  }
}

// The pool's ascending half-cleaner (graph_search.cuh:933-957): compare-
// exchanges at distances L/2 .. 1, in registers for distances >= 32.
template <int NL>
__device__ __forceinline__ void half_clean(float (&pd)[pool_regs(NL)], int (&pi)[pool_regs(NL)], int lane) {
  constexpr int L = pool_slots(NL), PR = pool_regs(NL);
#pragma unroll
  for (int rs = PR / 2; rs >= 1; rs >>= 1) {
#pragma unroll
    for (int j = 0; j < PR; ++j) {
      if (j & rs) continue;
      cx_regs(pd[j], pi[j], pd[j + rs], pi[j + rs], false);
    }
  }
  constexpr int kFirst = L < 32 ? L / 2 : 16;
  if constexpr (PR <= 2) {
#pragma unroll
    for (int sub = kFirst; sub >= 1; sub >>= 1) {
#pragma unroll
      for (int j = 0; j < PR; ++j) cx_lanes(pd[j], pi[j], sub, false, lane);
    }
  } else {
#pragma unroll 1
    for (int sub = kFirst; sub >= 1; sub >>= 1) {
#pragma unroll
      for (int j = 0; j < PR; ++j) cx_lanes(pd[j], pi[j], sub, false, lane);
    }
  }
}

// Pool/batch merge then the ascending half-cleaner (graph_search.cuh:921-957,
// :1454-1493).  Pool slot L-n+i meets batch slot B-n+i (n = min(L,B)); both
// are in the same lane.  The reference's main loop skips a batch slot holding
// MAX; a pool slot is never above MAX, so the strict comparison does too.
template <int NL, int NB>
__device__ __forceinline__ void merge_pool(float (&pd)[pool_regs(NL)], int (&pi)[pool_regs(NL)],
                                           const float (&bd)[batch_regs(NB)],
                                           const int (&bi)[batch_regs(NB)], int lane) {
  constexpr int PR = pool_regs(NL);
  auto meet = [&](int pr, bool mine, float od, int oi) {
    if (mine && pd[pr] > od) {
      pd[pr] = od;
      pi[pr] = oi;
    }
  };
  if constexpr (NB == 0) {
    // 16-slot batch: n = 16, batch slot i (lane i) meets pool slot L-16+i,
    // which is lane i of a 16-slot pool or lane 16+i of the last register
    float od = bd[0];
    int oi = bi[0];
    if constexpr (NL != 0) {
      od = __shfl_up_sync(kFull, od, 16);
      oi = __shfl_up_sync(kFull, oi, 16);
    }
    meet(PR - 1, NL == 0 ? lane < 16 : lane >= 16, od, oi);
  } else if constexpr (NL == 0) {
    // 16-slot pool: pool slot i (lane i) meets batch slot B-16+i, which is
    // lane 16+i of the last batch register.
    const float od = __shfl_down_sync(kFull, bd[NB - 1], 16);
    const int oi = __shfl_down_sync(kFull, bi[NB - 1], 16);
    meet(0, lane < 16, od, oi);
  } else {
    constexpr int NC = NL < NB ? NL : NB;
#pragma unroll
    for (int m = 0; m < NC; ++m) meet(NL - NC + m, true, bd[NB - NC + m], bi[NB - NC + m]);
  }
  half_clean<NL>(pd, pi, lane);
}

// ---- merging by rank ----
// A batch's candidates are the distances strictly below the pool's largest.
// When none is, the merge takes nothing -- it swaps only where pool > batch,
// and every pool slot is <= the largest -- and the half-cleaner then meets a
// pool that is still sorted ascending, where its strict comparisons swap
// nothing: the pool stays as it is, ids and order included.
//
// With m candidates whose distances are pairwise distinct, the descending
// batch sort puts them in the batch's last slots in descending order whatever
// the network does with the other slots: the candidate of ascending rank r
// lands in batch slot B-1-r, which the merge pairs with pool slot L-1-r.
// Every other batch slot holds a distance >= the pool's largest, so its
// comparison takes nothing.  Placing each candidate against pool slot L-1-r
// by its rank and running the half-cleaner (place_half_clean) therefore gives
// exactly the network's pool, ties with or within the pool included.  Anything
// else -- equal candidates, NaN, more candidates than kept -- runs the
// reference's network, where the handling of equal keys decides which id lands
// where.
//
// All of this needs a pool that is sorted ascending.  A batch with a NaN breaks
// that: no comparison with it swaps, so the batch sort, and then the pool, may
// come out in any order (a NaN itself never enters the pool, as pool > NaN is
// false).  From a query's first such batch that reaches the network on, all of
// its batches go through the network (kPoolUnsorted).  Checking the pool and
// going back once it is sorted again would serve only such queries, and cost
// the others: 10k queries at beam 256 and width 4 2.48 ms instead of 2.39.
//
// The candidates are compacted in shared memory and ranked one or two per
// lane against broadcast reads: about 2 instructions per candidate, where
// ranking them in the batch's slots by shuffles took 15 to 90, and no wide
// network in the usual case.  On one GB300 this took the 256-slot pools
// (10k queries, 500k x 96, BF16, beam 256, width 4) with the filter below from
// 3.80 to 2.5 ms.  Moving the pool's slots straight to their merged places, by
// comparing each candidate with the one register it falls into, was slower on
// bases of up to 1M rows, as its loop over the candidates is serial: 128 slots
// FP32 300 queries 416 / 321 us with the half-cleaner, 10k 2.63 / 2.24 ms; BF16
// 2,049 queries 576 / 512 us; 256 slots FP32 300 queries 498 / 357 us, BF16 10k
// 2.77 / 2.64 ms.  Over 10M x 96 it was slower for FP32 and FP8 rows (5.23 / 5.07
// and 5.78 / 5.41 ms at 256 slots, width 4), and for BF16 rows faster, 4.91 and
// 5.90 ms, where the half-cleaner takes 4.35 ms since those rows' loads are issued
// together (mma_group) and two warps share a query (team_floor).
template <int NL, int NB>
__host__ __device__ constexpr int cands_per_lane() { return batch_regs(NB) >= 4 ? 2 : 1; }
template <int NL, int NB>
__host__ __device__ constexpr int cand_limit() {
  constexpr int S = batch_slots(NB) > pool_slots(NL) ? batch_slots(NB) : pool_slots(NL);
  return S < 32 ? S : 32 * cands_per_lane<NL, NB>();
}

// Candidates that are inserted one by one instead of ranked (pools of one or
// two registers).
constexpr int kInsertMax = 4;
template <int NL>
__host__ __device__ constexpr bool inserts() { return pool_regs(NL) <= 2; }

// One candidate into the sorted pool; eq is set if a slot equals it.
template <int NL>
__device__ __forceinline__ void insert_one(float (&pd)[pool_regs(NL)], int (&pi)[pool_regs(NL)], float v, int id,
                                           bool& eq, int lane) {
  constexpr int PR = pool_regs(NL);
  float last_d = 0.0f;
  int last_i = 0;
#pragma unroll
  for (int j = 0; j < PR; ++j) {
    float up_d = __shfl_up_sync(kFull, pd[j], 1);
    int up_i = __shfl_up_sync(kFull, pi[j], 1);
    if (lane == 0) {
      up_d = j > 0 ? last_d : v;
      up_i = last_i;
    }
    if (j + 1 < PR) {
      last_d = __shfl_sync(kFull, pd[j], 31);
      last_i = __shfl_sync(kFull, pi[j], 31);
    }
    eq |= pd[j] == v;
    if (pd[j] > v && (NL != 0 || lane < 16)) {
      const bool moved = up_d > v;
      pd[j] = moved ? up_d : v;
      pi[j] = moved ? up_i : id;
    }
  }
}

// A search's loop state, in one register (a register of its own for the flag
// made kernels spill): the iterations since the visited filter's last rebuild,
// and whether the pool may be out of order.
constexpr int kRebuildAge = 7;    // mask of the count
constexpr int kPoolUnsorted = 8;  // a slot may be above the next one

// Merges the batch's candidates, (s_dist, s_ids)[0, n) below pmax, into a
// sorted pool, as far as that can be done here: none or a few inserted ones
// leave the pool done and give 0; otherwise they are compacted, ranked and left
// sorted ascending in slots [0, m), padded with +inf to a multiple of four, and
// m is returned; or -1, pool and arrays as they were, if the network has to run.
template <int NL, int NB>
__device__ __forceinline__ int rank_candidates(float (&pd)[pool_regs(NL)], int (&pi)[pool_regs(NL)], int* s_ids,
                                               float* s_dist, int n, float pmax, bool ties, int& state, int lane) {
  constexpr int PR = pool_regs(NL);
  constexpr int KC = cands_per_lane<NL, NB>();
  constexpr int kLim = cand_limit<NL, NB>();
  const unsigned lt = (1u << lane) - 1u;
  // the candidates of the first two blocks of 32, which hold most batches
  constexpr int NK = batch_regs(NB) < 2 ? 1 : 2;
  float d0[NK];
  unsigned c0[NK];
  int m = 0;
  bool nan = false;
#pragma unroll
  for (int t = 0; t < NK; ++t) {
    const int i = 32 * t + lane;
    d0[t] = i < n ? s_dist[i] : kMaxDist;
    c0[t] = __ballot_sync(kFull, d0[t] < pmax);
    nan |= d0[t] != d0[t];
    m += __popc(c0[t]);
  }
#pragma unroll 1
  for (int b = 32 * NK; b < n; b += 32) {
    const float d = b + lane < n ? s_dist[b + lane] : kMaxDist;
    nan |= d != d;
    m += __popc(__ballot_sync(kFull, d < pmax));
  }
  if (m == 0) return 0;
  if (__any_sync(kFull, nan)) {
    state |= kPoolUnsorted;
    return -1;
  }
  if constexpr (inserts<NL>()) {
    // One to four candidates are inserted one after the other: every slot
    // above the candidate moves up by one.  Without ties this is again the
    // one ascending order of the L smallest; with one, the pool is put back.
    if (m <= kInsertMax && !ties) {
      float sd[PR];
      int si[PR];
#pragma unroll
      for (int j = 0; j < PR; ++j) {
        sd[j] = pd[j];
        si[j] = pi[j];
      }
      bool eq = false;
#pragma unroll
      for (int t = 0; t < NK; ++t) {
        for (unsigned c = c0[t]; c; c &= c - 1) {
          const int src = __ffs(c) - 1;
          insert_one<NL>(pd, pi, __shfl_sync(kFull, d0[t], src), s_ids[32 * t + src], eq, lane);
        }
      }
#pragma unroll 1
      for (int b = 32 * NK; b < n; b += 32) {
        const float d = b + lane < n ? s_dist[b + lane] : kMaxDist;
        for (unsigned c = __ballot_sync(kFull, d < pmax); c; c &= c - 1) {
          const int src = __ffs(c) - 1;
          insert_one<NL>(pd, pi, __shfl_sync(kFull, d, src), s_ids[b + src], eq, lane);
        }
      }
      if (!__any_sync(kFull, eq)) return 0;
#pragma unroll
      for (int j = 0; j < PR; ++j) {
        pd[j] = sd[j];
        pi[j] = si[j];
      }
      return -1;
    }
  }
  if (m > kLim) return -1;
  // compact them, keeping the slots that this overwrites
  float od[KC];
  int oi[KC];
#pragma unroll
  for (int t = 0; t < KC; ++t) {
    const int i = 32 * t + lane;
    od[t] = i < n ? s_dist[i] : kMaxDist;
    oi[t] = i < n ? s_ids[i] : 0;
  }
  int at = 0;
#pragma unroll 1
  for (int b = 0; b < n; b += 32) {
    const int i = b + lane;
    const float d = i < n ? s_dist[i] : kMaxDist;
    const int id = i < n ? s_ids[i] : 0;
    const unsigned mask = __ballot_sync(kFull, d < pmax);
    __syncwarp();  // slots of this block and below have been read
    if (d < pmax) {
      s_dist[at + __popc(mask & lt)] = d;
      s_ids[at + __popc(mask & lt)] = id;
    }
    at += __popc(mask);
    __syncwarp();
  }
  bool ok;
  {
#pragma unroll
    for (int t = 0; t < KC; ++t) {
      const int i = 32 * t + lane;
      if (i >= m && i < kLim) s_dist[i] = __int_as_float(0x7f800000);
    }
    __syncwarp();
    float v[KC];
    int id[KC], r[KC];
#pragma unroll
    for (int t = 0; t < KC; ++t) {
      const int i = 32 * t + lane;
      v[t] = i < kLim ? s_dist[i] : 0.0f;
      id[t] = i < kLim ? s_ids[i] : 0;
      r[t] = 0;
    }
#pragma unroll 2
    for (int i = 0; i < m; i += 4) {
      const float4 w = *reinterpret_cast<const float4*>(s_dist + i);
#pragma unroll
      for (int t = 0; t < KC; ++t)
        r[t] += (w.x < v[t] ? 1 : 0) + (w.y < v[t] ? 1 : 0) + (w.z < v[t] ? 1 : 0) + (w.w < v[t] ? 1 : 0);
    }
    // distinct distances have distinct ranks
    int ranks = 0;
#pragma unroll
    for (int t = 0; t < KC; ++t) {
      unsigned bit[KC];
#pragma unroll
      for (int u = 0; u < KC; ++u) bit[u] = 32 * u + lane < m && (r[u] >> 5) == t ? 1u << (r[u] & 31) : 0u;
      unsigned all = bit[0];
      if constexpr (KC == 2) all |= bit[1];
      ranks += __popc(__reduce_or_sync(kFull, all));
    }
    ok = ranks == m;
    __syncwarp();
    if (ok) {
#pragma unroll
      for (int t = 0; t < KC; ++t)
        if (32 * t + lane < m) {
          s_dist[r[t]] = v[t];
          s_ids[r[t]] = id[t];
        }
    }
  }
  if (!ok) {
    __syncwarp();
#pragma unroll
    for (int t = 0; t < KC; ++t) {
      const int i = 32 * t + lane;
      if (i < n) {
        s_dist[i] = od[t];
        s_ids[i] = oi[t];
      }
    }
  }
  __syncwarp();
  return ok ? m : -1;
}

// Ranked candidate r against pool slot L-1-r, then the half-cleaner.
template <int NL, int NB>
__device__ __forceinline__ void place_half_clean(float (&pd)[pool_regs(NL)], int (&pi)[pool_regs(NL)],
                                                 const int* s_ids, const float* s_dist, int m, int lane) {
  constexpr int PR = pool_regs(NL);
#pragma unroll
  for (int t = 0; t < cands_per_lane<NL, NB>(); ++t) {
    const int r = 32 * t + (NL == 0 ? 15 : 31) - lane;
    if (t < PR && r >= 0 && r < m) {
      const float v = s_dist[r];
      if (pd[PR - 1 - (t < PR ? t : 0)] > v) {
        pd[PR - 1 - (t < PR ? t : 0)] = v;
        pi[PR - 1 - (t < PR ? t : 0)] = s_ids[r];
      }
    }
  }
  half_clean<NL>(pd, pi, lane);
}

// True when two neighbouring slots of the sorted pool hold equal distances
// of real points.
template <int NL>
__device__ __forceinline__ bool pool_has_ties(const float (&pd)[pool_regs(NL)], int lane) {
  constexpr int PR = pool_regs(NL);
  bool tie = false;
#pragma unroll
  for (int j = 0; j < PR; ++j) {
    float prev = __shfl_up_sync(kFull, pd[j], 1);
    if (j > 0) {
      const float last = __shfl_sync(kFull, pd[j > 0 ? j - 1 : 0], 31);
      if (lane == 0) prev = last;
    } else if (lane == 0) {
      prev = kMaxDist;
    }
    tie |= prev == pd[j] && pd[j] != kMaxDist;
  }
  return __any_sync(kFull, tie);
}

// Partial sum of one lane for one row: s = t0*t0, then fmaf(tc, tc, s) over
// chunks c (t = p - q on dims lane + 32c).  PREC selects the stored format;
// BF16 and FP8 rows are widened to FP32 before the subtraction.
template <int C, int PREC>
struct RowLoader;

template <int C>
struct RowLoader<C, kPrecF32> {
  float v[C];
  __device__ __forceinline__ void load(const SearchArgs& a, int id, int lane) {
    load_interleaved<C>(a.base + (size_t)id * (32 * C), lane, v);
  }
  __device__ __forceinline__ float value(int c) const { return v[c]; }
};

template <int C>
struct RowLoader<C, kPrecBF16> {
  float v[C];
  __device__ __forceinline__ void load(const SearchArgs& a, int id, int lane) {
    load_interleaved_bf16<C>(reinterpret_cast<const __nv_bfloat16*>(a.base_bf16) + (size_t)id * (32 * C), lane, v);
  }
  __device__ __forceinline__ float value(int c) const { return v[c]; }
};

template <int C>
struct RowLoader<C, kPrecFP8> {
  float v[C];
  __device__ __forceinline__ void load(const SearchArgs& a, int id, int lane) {
    float s = __ldg(a.fp8_scale + id);
    load_interleaved_fp8<C>(a.base_fp8 + (size_t)id * (32 * C), lane, v);
#pragma unroll
    for (int c = 0; c < C; ++c) v[c] *= s;
  }
  __device__ __forceinline__ float value(int c) const { return v[c]; }
};

template <int C>
__device__ __forceinline__ float lane_partial(const float (&p)[C], const float (&q)[C]) {
  float t = __fsub_rn(p[0], q[0]);
  float s = __fmul_rn(t, t);
#pragma unroll
  for (int c = 1; c < C; ++c) {
    t = __fsub_rn(p[c], q[c]);
    s = __fmaf_rn(t, t, s);
  }
  return s;
}

// ---- BF16 distances on the tensor cores (rows of 32*C <= 128 dims) ----
// A team: K warps of one block that serve one query (search_kernel_team).
// The leader (w == 0)
// runs the search; at each distance phase it publishes the row count in
// ctl[1] and the K warps each compute an interleaved share of the row groups
// into the leader's compaction buffers, between two crossings of the team's
// named barrier.  ctl[0] carries the team's query, ctl[1] = -1 ends it.
// Named barriers are hardware waits that every member reaches on every path,
// so a team needs no spin-wait.
struct Team {
  int K = 1;                     // warps per query
  int w = 0;                     // this warp's index in the team
  int bar = 0;                   // named barrier id (1 + team index in the block)
  volatile int* ctl = nullptr;   // [0] query, [1] phase: row count (+ 1<<16 for the rerank), -1 = done
};

__device__ __forceinline__ void team_sync(const Team& t) {
  asm volatile("bar.sync %0, %1;" ::"r"(t.bar), "r"(32 * t.K) : "memory");
}

// dist = |p|^2 + |q|^2 - 2 p.q, p the BF16 row, q the query rounded to BF16,
// p.q from mma.sync m16n8k16 (BF16 inputs, exact products, FP32
// accumulation).  A BF16 row (32*C values, 64*C bytes) is C pieces of 64
// interleaved bytes; thread t of each 4-thread group takes bytes
// [16t + 64i, +16) of piece i -- interleaved elements 32i + 8t + j, j < 8 --
// and uses them as the MMA k-slots {2t, 2t+1, 2t+8, 2t+9} of k-tiles 2i
// (j < 4) and 2i+1 (j >= 4).  In memory the bytes of two pieces lie side by
// side (bf16_offset), so one 256-bit load fetches both.
// The query fragment comes from the query's own BF16 row at the same
// interleaved positions, so each k pairs the base and query values of one
// dimension.
// With integer-valued data of magnitude < 2^8 every term is exact and the
// distances equal the FP32 path's bit for bit.
template <int C, int PREC, bool MMA = (PREC == kPrecBF16 && C >= 1 && C <= 4)>
struct QueryExtra {};
// Kernels for any chunk count (C == 0): the FP32 query row in the warp's
// shared memory, in the base rows' interleaved layout.
template <int PREC>
struct QueryExtra<0, PREC, false> {
  const float* qs;
};
template <int C, int PREC>
struct QueryExtra<C, PREC, true> {
  const uint32_t* qs;  // the query's BF16 row in the warp's shared memory (16*C words)
  float qn;            // squared norm of the BF16 query
};

__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                               uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The query in the base's BF16 layout, kept in `slot` (16*C words of the
// warp's shared memory) for the whole query, and its squared norm.
template <int C>
__device__ __forceinline__ void make_query_extra(QueryExtra<C, kPrecBF16, true>& qx,
                                                 const float (&qv)[C], uint32_t* slot, int lane) {
  uint16_t* qs = reinterpret_cast<uint16_t*>(slot);
  float s = 0.0f;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const __nv_bfloat16 b = __float2bfloat16_rn(qv[c]);
    const float f = __bfloat162float(b);
    s = __fmaf_rn(f, f, s);
    qs[interleaved_offset(c, lane, C)] = __bfloat16_as_ushort(b);
  }
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) s = __fadd_rn(s, __shfl_xor_sync(kFull, s, off));
  qx.qn = s;
  qx.qs = slot;
  __syncwarp();
}

// L2 prefetch of the rows a warp is about to gather, where the rows are too
// many to stay in L2 (SearchArgs::prefetch) and the warp has more than the
// one group of rows that it loads at once anyway.  On one GB300, prefetching
// always, or never: 10k queries over 96 MB of BF16 rows (beam 256, width 4)
// 2.54 and 2.47 ms; 2,049 queries over 256 MB (beam 128) 0.582 and 0.600 ms;
// one query as a team of 8 (one group a warp) 141 and 137 us.  A batch of up to
// kPrefetchWhole bytes is prefetched at once.  A larger one goes through a
// window of about kPrefetchBytes per warp: the first `ahead` rows of the
// warp's share before its first group, then at each group the rows `ahead`
// further on.  Without the window a batch of 256 rows of 3.8 KB would put
// ~1 MB per warp in flight, several GB over the grid against a 129 MB L2,
// and the lines would be evicted before use (on one GB300: 1.7x the
// algorithmic bytes read from DRAM).  Batches of up to 128 KB (256 FP32
// rows of 128 dims) measured faster prefetched whole.
constexpr int kPrefetchBytes = 16384;
constexpr int kPrefetchWhole = 196608;

__host__ __device__ constexpr int prefetch_ahead(int row_bytes, int G) {
  return kPrefetchBytes / row_bytes >= G ? kPrefetchBytes / row_bytes / G * G : G;
}
// Rows short enough that a batch of 256 is always prefetched whole: their
// kernels have no window code.
__host__ __device__ constexpr bool always_whole(int row_bytes) { return 256 * row_bytes <= kPrefetchWhole; }
// Rows to prefetch before the first group: all n, or the window.
__device__ __forceinline__ int prefetch_first(int n, int row_bytes, int ahead) {
  return n * row_bytes <= kPrefetchWhole ? n : ahead;
}

// Whether a member of a K-warp team prefetches at all.
__device__ __forceinline__ bool prefetch_pays(const SearchArgs& a, int n, int G, int K) {
  return a.prefetch && n > G * K;
}

// Prefetches rows [lr0, lr1) of member w's share of a K-warp team (groups
// of G rows, group g belonging to member g % K; a single warp is w = 0,
// K = 1), `lines` 128-byte lines per row.
template <int G>
__device__ __forceinline__ void prefetch_local(const char* rows, size_t row_bytes, int lines,
                                               const int* s_ids, int n, int lane, int w, int K, int lr0,
                                               int lr1) {
  // each lane keeps one line of every (32 / lines)-th row
  const int per = 32 / lines, r = lane / lines, line = lane - r * lines;
  if (r >= per) return;
  for (int lr = lr0 + r; lr < lr1; lr += per) {
    const int j = lr / G;
    const int row = G * (w + j * K) + (lr - j * G);
    if (row >= n) break;
    asm volatile("prefetch.global.L2 [%0];" ::"l"(rows + (size_t)s_ids[row] * row_bytes + line * 128));
  }
}

// Distances of the n ids in s_ids[0..n) by the tensor cores, 8 rows per MMA
// group: thread (g, t) supplies row g of the group as column g of the MMA's
// B operand; the query is every row of A, so every lane of thread index t
// holds the dot products of rows 2t and 2t+1: lane (0, t) finishes row 2t and
// lane (1, t) row 2t+1, with one norm load and one store each.
//
// The LSU's wavefronts bound the 10k-query batches (85 % of its peak in ncu
// on one GB300, 63 % issue).  A group of 8 rows of 128 dims took about 58:
// 32 for four 16-byte loads over half of 8 lines each, 8 + 2 for the norms
// and their ids, up to 16 for the query's fragments, 16 for its L2 prefetch.
// 256-bit loads make the first 16.
__device__ __forceinline__ void ldg256(const void* p, uint4& a, uint4& b) {
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
      : "l"(p));
}

// One group of 8 rows from r0 (rows >= n are skipped).
template <int C>
__device__ __forceinline__ void mma_group(const SearchArgs& a, const QueryExtra<C, kPrecBF16, true>& qx,
                                          const int* s_ids, float* s_dist, int n, int lane, int r0) {
  constexpr int kRowBytes = 64 * C;
  const char* rows = reinterpret_cast<const char*>(a.base_bf16);
  const int g = lane >> 2, t = lane & 3;
  // Rows of 4 chunks take the query's fragments ahead of the rows, shorter ones
  // as the MMAs need them, which leaves the compiler the registers to issue a
  // row's loads together.  One GB300, ahead / as needed: 10k queries over 1M x
  // 128 (beam 16) 487 / 519 us; over 500k x 96 (beam 256, width 4) 2.42 / 2.08 ms,
  // over 10M x 96 (beam 64) 1.79 / 1.53 ms.
  constexpr bool kQueryAhead = C >= 4;
  uint4 qf[C];
  if constexpr (kQueryAhead) {
#pragma unroll
    for (int i = 0; i < C; ++i) qf[i] = *reinterpret_cast<const uint4*>(qx.qs + 4 * t + 16 * i);
  }
  const int id = s_ids[r0 + g < n ? r0 + g : r0];
  const char* p = rows + (size_t)id * kRowBytes;
  uint4 v[C];
  if constexpr (bf16_paired(C)) {
#pragma unroll
    for (int i = 0; i + 1 < C; i += 2) ldg256(p + 64 * i + 32 * t, v[i], v[i + 1]);
    if constexpr (C & 1) v[C - 1] = __ldg(reinterpret_cast<const uint4*>(p + 64 * (C - 1) + 16 * t));
  } else {
#pragma unroll
    for (int i = 0; i < C; ++i) v[i] = __ldg(reinterpret_cast<const uint4*>(p + 64 * i + 16 * t));
  }
  // the norm of the row this lane finishes, loaded while the MMAs run
  const int row = r0 + 2 * t + g;
  const bool mine = g < 2 && row < n;
  const float pn = mine ? __ldg(a.norm16 + s_ids[row]) : 0.0f;
  float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int i = 0; i < C; ++i) {
    if constexpr (!kQueryAhead) qf[i] = *reinterpret_cast<const uint4*>(qx.qs + 4 * t + 16 * i);
    mma_bf16_16816(d, qf[i].x, qf[i].x, qf[i].y, qf[i].y, v[i].x, v[i].y);
    mma_bf16_16816(d, qf[i].z, qf[i].z, qf[i].w, qf[i].w, v[i].z, v[i].w);
  }
  if (mine) s_dist[row] = __fmaf_rn(-2.0f, g == 0 ? d[0] : d[1], __fadd_rn(pn, qx.qn));
}

template <int C, bool TEAM>
__device__ __forceinline__ void distances_mma(const SearchArgs& a, const QueryExtra<C, kPrecBF16, true>& qx,
                                              const int* s_ids, float* s_dist, int n, int lane, int w, int K) {
  constexpr int kRowBytes = 64 * C, kLines = (kRowBytes + 127) / 128;
  static_assert(always_whole(kRowBytes), "no prefetch window");
  const char* rows = reinterpret_cast<const char*>(a.base_bf16);
  const int ws = TEAM ? w : 0, ks = TEAM ? K : 1;
  if (prefetch_pays(a, n, 8, ks)) prefetch_local<8>(rows, kRowBytes, kLines, s_ids, n, lane, ws, ks, 0, n);
#pragma unroll 1
  for (int r0 = 8 * ws; r0 < n; r0 += 8 * ks) mma_group<C>(a, qx, s_ids, s_dist, n, lane, r0);
}

// ---- rows of a run-time chunk count (kernels built for any dimension) ----
// A row of C chunks is streamed slab by slab in the interleaved layout
// (layout.cuh): chunks 4s..4s+3 as one 4-value load per lane, then a pair,
// then a single chunk.  Each value is widened to FP32 (BF16 exactly; FP8
// times the row's scale) before the subtraction, as RowLoader does.  A slab's
// loads of all rows of a group come first, as raw bytes, and are widened row by
// row (rt_group): widened at the load, BF16 rows took 16 registers instead of 8
// and the compiler put the loads of some kernels one after the other.  One GB300,
// one warp per query: 40k x 512, degree 64, beam 64, 10k queries 5.7 ms so, 3.7
// ms now; 80k x 256 4.2 and 3.1 ms.
template <int PREC>
struct SlabLoader;

template <>
struct SlabLoader<kPrecF32> {
  const float* row;
  __device__ __forceinline__ void init(const SearchArgs& a, int id, size_t stride) { row = a.base + (size_t)id * stride; }
  using Raw = float4;
  __device__ __forceinline__ Raw quad_raw(int off, int lane) const {
    return __ldg(reinterpret_cast<const float4*>(row + off) + lane);
  }
  __device__ __forceinline__ float4 widen4(const Raw& x) const { return x; }
  __device__ __forceinline__ float2 pair(int off, int lane) const {
    return __ldg(reinterpret_cast<const float2*>(row + off) + lane);
  }
  __device__ __forceinline__ float one(int off, int lane) const { return __ldg(row + off + lane); }
};

template <>
struct SlabLoader<kPrecBF16> {
  const uint16_t* row;
  int C;
  __device__ __forceinline__ void init(const SearchArgs& a, int id, size_t stride) {
    row = a.base_bf16 + (size_t)id * stride;
    C = a.C;
  }
  // Rows of 2 to 4 chunks are stored in the paired layout (bf16_offset): their
  // one slab of four chunks, or the pair, starts the row, and a last odd chunk
  // is not moved.
  using Raw = uint2;
  __device__ __forceinline__ Raw quad_raw(int off, int lane) const {
    const int at = C == 4 ? bf16_offset(4 * lane, 4) : 4 * lane;
    return __ldg(reinterpret_cast<const uint2*>(row + off + at));
  }
  __device__ __forceinline__ float4 widen4(const Raw& x) const {
    return make_float4(bf16lo(x.x), bf16hi(x.x), bf16lo(x.y), bf16hi(x.y));
  }
  __device__ __forceinline__ float2 pair(int off, int lane) const {
    const int at = C < 4 ? bf16_offset(2 * lane, 3) : 2 * lane;
    const uint32_t y = __ldg(reinterpret_cast<const unsigned int*>(row + off + at));
    return make_float2(bf16lo(y), bf16hi(y));
  }
  __device__ __forceinline__ float one(int off, int lane) const {
    return __uint_as_float((uint32_t)__ldg(row + off + lane) << 16);
  }
};

template <>
struct SlabLoader<kPrecFP8> {
  const uint8_t* row;
  float sc;
  __device__ __forceinline__ void init(const SearchArgs& a, int id, size_t stride) {
    row = a.base_fp8 + (size_t)id * stride;
    sc = __ldg(a.fp8_scale + id);
  }
  using Raw = uint32_t;
  __device__ __forceinline__ Raw quad_raw(int off, int lane) const {
    return __ldg(reinterpret_cast<const unsigned int*>(row + off) + lane);
  }
  __device__ __forceinline__ float4 widen4(const Raw& x) const {
    const float2 u = fp8x2_to_float2((uint16_t)(x & 0xffffu));
    const float2 v = fp8x2_to_float2((uint16_t)(x >> 16));
    return make_float4(__fmul_rn(u.x, sc), __fmul_rn(u.y, sc), __fmul_rn(v.x, sc), __fmul_rn(v.y, sc));
  }
  __device__ __forceinline__ float2 pair(int off, int lane) const {
    const float2 u = fp8x2_to_float2(__ldg(reinterpret_cast<const unsigned short*>(row + off) + lane));
    return make_float2(__fmul_rn(u.x, sc), __fmul_rn(u.y, sc));
  }
  __device__ __forceinline__ float one(int off, int lane) const {
    return __fmul_rn(fp8x2_to_float2((uint16_t)__ldg(row + off + lane)).x, sc);
  }
};

// One chunk of a lane's partial: fmaf(t, t, s) with t = p - q.  The first
// chunk starts from s = +0, and fmaf(t, t, +0) rounds exactly as t * t, so
// the sum equals lane_partial's.
__device__ __forceinline__ float chunk_acc(float p, float q, float s) {
  const float t = __fsub_rn(p, q);
  return __fmaf_rn(t, t, s);
}

// The butterfly reduction of G rows' lane partials (see `distances`): row
// g0 + lane / (32/G) is complete in the first lane of each 32/G-lane span.
template <int G>
__device__ __forceinline__ void reduce_rows(float (&part)[G], float* s_dist, int g0, int n, int lane) {
  constexpr int SPAN = 32 / G;
#pragma unroll
  for (int off = 16, half = G / 2; half >= 1; off >>= 1, half >>= 1) {
    const bool up = (lane & off) != 0;
#pragma unroll
    for (int t = 0; t < half; ++t) {
      float send = up ? part[t] : part[t + half];
      float keep = up ? part[t + half] : part[t];
      part[t] = __fadd_rn(keep, __shfl_xor_sync(kFull, send, off));
    }
  }
  float total = part[0];
#pragma unroll
  for (int off = SPAN / 2; off >= 1; off >>= 1) total = __fadd_rn(total, __shfl_xor_sync(kFull, total, off));
  const int row = g0 + lane / SPAN;
  if ((lane % SPAN) == 0 && row < n) s_dist[row] = total;
}

// Distances of n rows of a.C chunks against the query row in shared memory
// qs (interleaved layout), G rows in flight.
// One group of 4 rows from g0 of a run-time chunk count (rows >= n give 0).
template <int PREC>
__device__ __forceinline__ void rt_group(const SearchArgs& a, const float* qs, const int* s_ids,
                                         float* s_dist, int n, int lane, int g0) {
  constexpr int G = 4;
  const int C = a.C, n4 = C >> 2, rem = C & 3;
  const size_t stride = 32 * (size_t)C;  // elements per row
  SlabLoader<PREC> r[G];
#pragma unroll
  for (int t = 0; t < G; ++t) r[t].init(a, s_ids[g0 + t < n ? g0 + t : g0], stride);
  float part[G];
#pragma unroll
  for (int t = 0; t < G; ++t) part[t] = 0.0f;
#pragma unroll 2
  for (int sl = 0; sl < n4; ++sl) {
    typename SlabLoader<PREC>::Raw raw[G];
#pragma unroll
    for (int t = 0; t < G; ++t) raw[t] = r[t].quad_raw(128 * sl, lane);
    const float4 q = *reinterpret_cast<const float4*>(qs + 128 * sl + 4 * lane);
#pragma unroll
    for (int t = 0; t < G; ++t) {
      const float4 v = r[t].widen4(raw[t]);
      part[t] = chunk_acc(v.x, q.x, part[t]);
      part[t] = chunk_acc(v.y, q.y, part[t]);
      part[t] = chunk_acc(v.z, q.z, part[t]);
      part[t] = chunk_acc(v.w, q.w, part[t]);
    }
  }
  int off = 128 * n4;
  if (rem >= 2) {
    const float2 q = *reinterpret_cast<const float2*>(qs + off + 2 * lane);
#pragma unroll
    for (int t = 0; t < G; ++t) {
      const float2 v = r[t].pair(off, lane);
      part[t] = chunk_acc(v.x, q.x, part[t]);
      part[t] = chunk_acc(v.y, q.y, part[t]);
    }
    off += 64;
  }
  if (rem & 1) {
    const float q = qs[off + lane];
#pragma unroll
    for (int t = 0; t < G; ++t) part[t] = chunk_acc(r[t].one(off, lane), q, part[t]);
  }
#pragma unroll
  for (int t = 0; t < G; ++t)
    if (g0 + t >= n) part[t] = 0.0f;
  reduce_rows<G>(part, s_dist, g0, n, lane);
}

template <int PREC>
__host__ __device__ constexpr int slab_bytes() {
  return PREC == kPrecF32 ? 4 : PREC == kPrecBF16 ? 2 : 1;
}

template <int PREC>
__device__ __forceinline__ const char* search_rows(const SearchArgs& a) {
  return PREC == kPrecF32    ? reinterpret_cast<const char*>(a.base)
         : PREC == kPrecBF16 ? reinterpret_cast<const char*>(a.base_bf16)
                             : reinterpret_cast<const char*>(a.base_fp8);
}

template <int PREC, bool TEAM>
__device__ __forceinline__ void distances_rt(const SearchArgs& a, const float* qs, const int* s_ids,
                                             float* s_dist, int n, int lane, int w, int K) {
  constexpr int G = 4;
  const size_t rb = 32 * (size_t)a.C * slab_bytes<PREC>();
  const int lines = (int)((rb + 127) / 128);
  const char* rows = search_rows<PREC>(a);
  const int ws = TEAM ? w : 0, ks = TEAM ? K : 1;
  const int ahead = prefetch_ahead((int)rb, G);
  const int first_rows = prefetch_first(n, (int)rb, ahead);
  const bool pays = prefetch_pays(a, n, G, ks);
  if (pays) prefetch_local<G>(rows, rb, lines, s_ids, n, lane, ws, ks, 0, first_rows);
  const bool windowed = pays && first_rows < n;
  const int first = G * ws, step = G * ks;
  int j = 0;
  for (int g0 = first; g0 < n; g0 += step, ++j) {
    if (windowed) prefetch_local<G>(rows, rb, lines, s_ids, n, lane, ws, ks, ahead + G * j, ahead + G * j + G);
    rt_group<PREC>(a, qs, s_ids, s_dist, n, lane, g0);
  }
}

// Distances of the n (<= B) ids in s_ids[0..n) written to s_dist[0..n).
// Groups of G rows (16, or 8 for long rows): each lane forms its partial for
// the G rows; a butterfly over offsets 16, 8, ... exchanges half of the rows
// at each level until every lane holds one row, then plain xor-shuffles
// finish the sum, which lands in the 32/G lanes lane = t*(32/G) + ...
// Every addition pairs the same two partial sums as the reference's
// shuffle-down tree (addition is commutative, so the results are equal).
// With TEAM, the groups of rows of member w of a K-warp team only.
// Rows per distance group of each path.
template <int C, int PREC>
__host__ __device__ constexpr int distance_group_size() {
  return C == 0 ? 4 : (PREC == kPrecBF16 && C <= 4) ? 8 : C <= 4 ? 8 : 2;
}

// One group of rows with the query in registers (C > 0, scalar path): all
// G loads first, unconditionally (a short group re-reads its first row), so
// they are issued back to back before any use.
template <int C, int PREC>
__device__ __forceinline__ void regs_group(const SearchArgs& a, const float (&qv)[qregs(C)], const int* s_ids,
                                           float* s_dist, int n, int lane, int g0) {
  constexpr int G = distance_group_size<C, PREC>();
  RowLoader<C, PREC> r[G];
#pragma unroll
  for (int t = 0; t < G; ++t) r[t].load(a, s_ids[g0 + t < n ? g0 + t : g0], lane);
  float part[G];
#pragma unroll
  for (int t = 0; t < G; ++t) part[t] = g0 + t < n ? lane_partial<C>(r[t].v, qv) : 0.0f;
  reduce_rows<G>(part, s_dist, g0, n, lane);
}

// Group `grp` (rows grp*G ..) of a batch, on whichever path the kernel uses.
template <int C, int PREC>
__device__ __forceinline__ void distance_group(const SearchArgs& a, const float (&qv)[qregs(C)],
                                               const QueryExtra<C, PREC>& qx, const int* s_ids,
                                               float* s_dist, int n, int lane, int grp) {
  constexpr int G = distance_group_size<C, PREC>();
  if constexpr (C == 0)
    rt_group<PREC>(a, qx.qs, s_ids, s_dist, n, lane, G * grp);
  else if constexpr (PREC == kPrecBF16 && C <= 4)
    mma_group<C>(a, qx, s_ids, s_dist, n, lane, G * grp);
  else
    regs_group<C, PREC>(a, qv, s_ids, s_dist, n, lane, G * grp);
}

// The L2 prefetch a batch's distances start with (the whole batch, or the
// first window of a large one), for a warp that computes any of its groups.
template <int C, int PREC>
__device__ __forceinline__ void prefetch_batch(const SearchArgs& a, const int* s_ids, int n, int lane) {
  constexpr int G = distance_group_size<C, PREC>();
  const int rb = 32 * (C == 0 ? a.C : C) * slab_bytes<PREC>();
  const int lines = (rb + 127) / 128;
  if (prefetch_pays(a, n, G, 1))
    prefetch_local<G>(search_rows<PREC>(a), rb, lines, s_ids, n, lane, 0, 1, 0,
                      prefetch_first(n, rb, prefetch_ahead(rb, G)));
}

// ---- helping in the tail ----
// When the query counter runs out, the warps left without a query help the
// warps of their block still searching: a leader with idle warps in its
// block publishes each batch's distance phase, and leader and helpers take
// its groups of rows from one ticket.  Every row's arithmetic is the
// leader's own, so results are unchanged.  While no warp of the block is
// idle (all but the last queries) a leader only reads the idle count.
struct PhaseDesc {
  unsigned long long ticket;  // (generation << 32) | next group to take
  unsigned long long gen_n;   // (generation << 32) | rows of the phase, one word
  int q;                      // the phase's query
  float qn;                   // its BF16 squared norm (tensor-core distances)
  int done;                   // groups finished by helpers
  int pad;
};
struct BlockShare {
  unsigned int idle;          // warps of the block with no query left
  unsigned int pad[3];
  PhaseDesc desc[8];
};
static_assert(sizeof(BlockShare) == kBlockShareBytes, "block share layout");

// The kernels that help in the tail: the tensor-core BF16 rows and the rows
// of any chunk count, with batches of up to 64 slots.  The scalar register
// path (FP32 and FP8 rows of up to 4 chunks, and 30 chunks) holds a group of
// rows in registers, and a second copy of it for the helped phase made those
// kernels spill at 64 registers.  Batches of 128 and 256 slots measured
// slower helped (one ticket per group of 8 rows over 16-32 groups).
template <int C, int PREC, int NB>
__host__ __device__ constexpr bool tail_helping() {
  return (C == 0 || (PREC == kPrecBF16 && C >= 1 && C <= 4)) && NB <= 2;
}

constexpr long long kHelpWaitLimit = 1ll << 24;   // leader's polls for helpers' groups
constexpr long long kHelperIdleLimit = 1ll << 21; // empty scans (~0.4 s) before a helper leaves

// The block's share, after its warps' regions (per_warp words each; a
// multiple of 4, so 16-byte aligned).
__device__ __forceinline__ BlockShare* block_share(uint32_t* smem, int per_warp) {
  return reinterpret_cast<BlockShare*>(smem + (size_t)(blockDim.x >> 5) * per_warp);
}

// The leader's side of a helped distance phase.  Publishes (q, qn, n) and
// the generation, takes groups from the ticket, then waits for the groups
// helpers took (bounded; on timeout the error word is set).
template <int C, int PREC>
__device__ __forceinline__ void helped_distances(const SearchArgs& a, const float (&qv)[qregs(C)],
                                                 const QueryExtra<C, PREC>& qx, const int* s_ids,
                                                 float* s_dist, int n, int lane, int q, float qn,
                                                 BlockShare* bs) {
  constexpr int G = distance_group_size<C, PREC>();
  PhaseDesc& d = bs->desc[threadIdx.x >> 5];
  const int ng = (n + G - 1) / G;
  if (lane == 0) {
    const unsigned gen = (unsigned)(*reinterpret_cast<volatile unsigned long long*>(&d.gen_n) >> 32) + 1u;
    d.q = q;
    d.qn = qn;
    d.done = 0;
    *reinterpret_cast<volatile unsigned long long*>(&d.gen_n) = ((unsigned long long)gen << 32) | (unsigned)n;
    __threadfence_block();
    atomicExch(&d.ticket, (unsigned long long)gen << 32);
  }
  __syncwarp();
  prefetch_batch<C, PREC>(a, s_ids, n, lane);
  int mine = 0;
  for (;;) {
    unsigned long long old = 0;
    if (lane == 0) old = atomicAdd(&d.ticket, 1ull);
    const int grp = (int)__shfl_sync(kFull, (unsigned)old, 0);
    if (grp >= ng) break;
    distance_group<C, PREC>(a, qv, qx, s_ids, s_dist, n, lane, grp);
    ++mine;
  }
  if (lane == 0) {
    const int expect = ng - mine;  // every group below ng was taken by someone
    long long it = 0;
    while (*reinterpret_cast<volatile int*>(&d.done) < expect) {
      if (++it > kHelpWaitLimit) {
        if (a.err) atomicExch(a.err, kErrHelpWait);
        break;
      }
    }
    __threadfence_block();
  }
  __syncwarp();
}

template <int C, int PREC, bool TEAM = false>
__device__ __forceinline__ void distances(const SearchArgs& a, const float (&qv)[qregs(C)],
                                          const QueryExtra<C, PREC>& qx, const int* s_ids,
                                          float* s_dist, int n, int lane, int w = 0, int K = 1) {
  if constexpr (C == 0) {
    distances_rt<PREC, TEAM>(a, qx.qs, s_ids, s_dist, n, lane, w, K);
  } else if constexpr (PREC == kPrecBF16 && C <= 4) {
    distances_mma<C, TEAM>(a, qx, s_ids, s_dist, n, lane, w, K);
  } else {
    constexpr int G = C <= 4 ? 8 : 2;
    constexpr int kRowBytes = 32 * C * (PREC == kPrecF32 ? 4 : PREC == kPrecBF16 ? 2 : 1);
    constexpr int kLines = (kRowBytes + 127) / 128, kAhead = prefetch_ahead(kRowBytes, G);
    const char* rows = PREC == kPrecF32    ? reinterpret_cast<const char*>(a.base)
                       : PREC == kPrecBF16 ? reinterpret_cast<const char*>(a.base_bf16)
                                           : reinterpret_cast<const char*>(a.base_fp8);
    const int ws = TEAM ? w : 0, ks = TEAM ? K : 1;
    const int first_rows = prefetch_first(n, kRowBytes, kAhead);
    const bool pays = prefetch_pays(a, n, G, ks);
    if (pays) prefetch_local<G>(rows, kRowBytes, kLines, s_ids, n, lane, ws, ks, 0, first_rows);
    const int first = G * ws, step = G * ks;
    auto group = [&](int g0) { regs_group<C, PREC>(a, qv, s_ids, s_dist, n, lane, g0); };
    // the window's loop is a copy of its own: the whole-batch loop keeps no
    // window state in the registers these rows fill
    if (always_whole(kRowBytes) || !pays || first_rows >= n) {
#pragma unroll 1
      for (int g0 = first; g0 < n; g0 += step) group(g0);
    } else {
      int j = 0;
      for (int g0 = first; g0 < n; g0 += step, ++j) {
        prefetch_local<G>(rows, kRowBytes, kLines, s_ids, n, lane, ws, ks, kAhead + G * j, kAhead + G * j + G);
        group(g0);
      }
    }
  }
}

// Appends the valid ids (0 <= id < np) of batch register j to the n ids in
// s_ids, in slot order, and returns their new number; lane j keeps the
// register's mask of valid slots in `slots`.
__device__ __forceinline__ int compact_slot(int np, int id, int j, int n, int* s_ids, unsigned& slots, int lane) {
  const bool v = id >= 0 && id < np;
  const unsigned m = __ballot_sync(kFull, v);
  if (v) s_ids[n + __popc(m & ((1u << lane) - 1u))] = id;
  if (lane == j) slots = m;
  return n + __popc(m);
}

// Distances of the n compacted ids in s_ids into s_dist.
// With TEAM, the team's warps share the distances (team leader only).
// Alone (not TEAM), with bs, idle warps of the block may help (tail).
template <int C, int NB, int PREC, bool TEAM = false>
__device__ __forceinline__ void batch_distances(const SearchArgs& a, const float (&qv)[qregs(C)],
                                                const QueryExtra<C, PREC>& qx, const int* s_ids,
                                                float* s_dist, int n, int lane, const Team& t = Team(),
                                                int q = 0, BlockShare* bs = nullptr) {
  if constexpr (TEAM) {
    if (lane == 0) t.ctl[1] = n;
    team_sync(t);
    distances<C, PREC, true>(a, qv, qx, s_ids, s_dist, n, lane, 0, t.K);
    team_sync(t);
  } else {
    __syncwarp();
    constexpr int G = distance_group_size<C, PREC>();
    if (tail_helping<C, PREC, NB>() && bs && n > G && *reinterpret_cast<volatile unsigned*>(&bs->idle) != 0u) {
      float qn = 0.0f;
      if constexpr (PREC == kPrecBF16 && C >= 1 && C <= 4) qn = qx.qn;
      if constexpr (tail_helping<C, PREC, NB>()) helped_distances<C, PREC>(a, qv, qx, s_ids, s_dist, n, lane, q, qn, bs);
    } else {
      distances<C, PREC>(a, qv, qx, s_ids, s_dist, n, lane);
    }
    __syncwarp();
  }
}

// The reference's merge of a batch held compacted in (s_ids, s_dist): the
// batch back in its slots (invalid ones hold MAX), sorted and merged by the
// network.
template <int NL, int NB>
__device__ __forceinline__ void merge_network(float (&pd)[pool_regs(NL)], int (&pi)[pool_regs(NL)], int np,
                                              const int* s_ids, const float* s_dist, unsigned slots,
                                              int lane) {
  constexpr int BR = batch_regs(NB);
  const unsigned lt = (1u << lane) - 1u;
  float bd[BR];
  int bi[BR];
  int at = 0;
#pragma unroll
  for (int j = 0; j < BR; ++j) {
    const unsigned m = __shfl_sync(kFull, slots, j);
    const bool v = (m >> lane) & 1u;
    const int k = at + __popc(m & lt);
    bd[j] = v ? s_dist[k] : kMaxDist;
    bi[j] = v ? s_ids[k] : np;
    at += __popc(m);
  }
  __syncwarp();
  sort_batch_desc<BR, true, batch_slots(NB)>(bd, bi, lane);
  merge_pool<NL, NB>(pd, pi, bd, bi, lane);
}

// The pool after a batch of n distances (compacted in s_ids / s_dist), m of
// them ranked candidates (rank_candidates; -1: the network).  `ties` says
// that two slots of the pool may be equal.
template <int NL, int NB>
__device__ __forceinline__ void merge_batch(float (&pd)[pool_regs(NL)], int (&pi)[pool_regs(NL)], int np,
                                            int* s_ids, float* s_dist, int m, unsigned slots, bool& ties,
                                            int lane) {
  if (m == 0) return;
  if (m > 0)
    place_half_clean<NL, NB>(pd, pi, s_ids, s_dist, m, lane);
  else
    merge_network<NL, NB>(pd, pi, np, s_ids, s_dist, slots, lane);
  __syncwarp();
  if constexpr (inserts<NL>()) ties = pool_has_ties<NL>(pd, lane);
}

// Exact FP32 rerank of the final pool for the reduced-precision paths: the
// pool ids (visited marks dropped) get FP32 distances computed exactly as
// the FP32 path computes them, then the pool is bitonic-sorted ascending.
// The reference's precedent is the host-side parallel_reorder
// (graph_helper.cu:146-213), which recomputes FP32 L2 and std::sorts.
template <int C, int NL, bool TEAM = false>
__device__ __forceinline__ void rerank_pool(const SearchArgs& a, const float (&qv)[qregs(C)],
                                            const float* qsm, float (&pd)[pool_regs(NL)],
                                            int (&pi)[pool_regs(NL)], int* s_ids, float* s_dist,
                                            int lane, const Team& t = Team()) {
  constexpr int PR = pool_regs(NL);
  const unsigned lt = (1u << lane) - 1u;
  unsigned slots = 0;  // lane j: the valid slots of pool register j
  int n = 0;
#pragma unroll
  for (int j = 0; j < PR; ++j) {
    const int id = pi[j] < 0 ? -pi[j] : pi[j];
    const bool v = id < a.np;
    const unsigned m = __ballot_sync(kFull, v);
    if (v) s_ids[n + __popc(m & lt)] = id;
    if (lane == j) slots = m;
    n += __popc(m);
  }
  QueryExtra<C, kPrecF32> q32{};
  if constexpr (C == 0) q32.qs = qsm;
  if constexpr (TEAM) {
    if (lane == 0) t.ctl[1] = n | (1 << 16);
    team_sync(t);
    distances<C, kPrecF32, true>(a, qv, q32, s_ids, s_dist, n, lane, 0, t.K);
    team_sync(t);
  } else {
    __syncwarp();
    distances<C, kPrecF32>(a, qv, q32, s_ids, s_dist, n, lane);
    __syncwarp();
  }
  int at = 0;
#pragma unroll
  for (int j = 0; j < PR; ++j) {
    const unsigned m = __shfl_sync(kFull, slots, j);
    const bool v = (m >> lane) & 1u;
    const int k = at + __popc(m & lt);
    pd[j] = v ? s_dist[k] : kMaxDist;
    pi[j] = v ? s_ids[k] : a.np;
    at += __popc(m);
  }
  __syncwarp();
  sort_batch_desc<PR, false, pool_slots(NL)>(pd, pi, lane);
}

// One query.  Batch slot p (lane p % 32 of register p / 32) belongs to the
// (p / R)-th node selected in the iteration and holds entry p % R of its
// neighbour list.  For R >= 32 a node's list fills R / 32 whole registers
// (register j holds node j / (R / 32)); R16 kernels serve degree-16 graphs,
// whose lists fill half a register (slot p holds node p / 16).
// The query's registers and shared-memory slot: FP32 chunks in registers
// (C > 0; plus its BF16 row in q_slot for the tensor-core distances), or the
// FP32 row in q_slot in the base's interleaved layout (C == 0).
template <int C>
__device__ __forceinline__ void load_query_chunks(const SearchArgs& a, int q, int lane, float (&qv)[qregs(C)]) {
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int dim = lane + 32 * c;
    qv[c] = dim < a.d ? __ldg(a.queries + (size_t)q * a.qstride + dim) : 0.0f;
  }
}

template <int C, int PREC>
__device__ __forceinline__ void load_query(const SearchArgs& a, int q, int lane, float (&qv)[qregs(C)],
                                           QueryExtra<C, PREC>& qx, uint32_t* q_slot) {
  if constexpr (C == 0) {
    float* qs = reinterpret_cast<float*>(q_slot);
    for (int c = 0; c < a.C; ++c) {
      const int dim = lane + 32 * c;
      qs[interleaved_offset(c, lane, a.C)] = dim < a.d ? __ldg(a.queries + (size_t)q * a.qstride + dim) : 0.0f;
    }
    qv[0] = 0.0f;
    qx.qs = qs;
    __syncwarp();
  } else {
    load_query_chunks<C>(a, q, lane, qv);
    if constexpr (PREC == kPrecBF16 && C <= 4) make_query_extra<C>(qx, qv, q_slot, lane);
  }
}

template <int C, int NL, int NB, int PREC, bool R16, bool TEAM = false>
__device__ __forceinline__ void search_query(const SearchArgs& a, int q, int lane, const Bloom& bloom,
                                             int* s_ids, float* s_dist, uint32_t* q_slot,
                                             const Team& t = Team(), BlockShare* bs = nullptr) {
  constexpr int L = pool_slots(NL);
  constexpr int PR = pool_regs(NL);  // pool registers
  constexpr int BR = batch_regs(NB);  // batch registers
  constexpr int B = batch_slots(NB);
  static_assert(R16 || NB > 0, "a 16-slot batch comes from a degree-16 graph");
  const int np = a.np;
  const int R = R16 ? 16 : a.R;
  const int NR = R >> 5;               // batch registers per node (R >= 32)
  const int nr_shift = __ffs(NR) - 1;  // j / NR == j >> nr_shift
  int c_entries = 0, c_expanded = 0, c_dists = 0;  // per query: far below 2^31

  float qv[qregs(C)];
  QueryExtra<C, PREC> qx;
  load_query<C, PREC>(a, q, lane, qv, qx, q_slot);

  float pd[PR];
  int pi[PR];
#pragma unroll
  for (int j = 0; j < PR; ++j) {
    pd[j] = kMaxDist;
    pi[j] = np;
  }
  unsigned slots = 0;  // lane j: the valid slots of batch register j
  bool ties = false;   // two pool slots may hold equal distances (merge_batch)

  bloom.clear(lane);
  __syncwarp();

  // ---- main loop state (graph_search.cuh:961-1532) ----
  uint32_t tmp_flag = L >= 32 ? 0xFFFFFFFFu : ((1u << L) - 1u);  // (1 << min(L,32)) - 1 (:969)
  int iteration = 0;
  bool cz = false;  // this lane's check_zero (:967)
  int state = 0;  // kRebuildAge and kPoolUnsorted
  int iter = 0;

  auto scan = [&](int chunk) -> uint32_t {  // :1019-1028, :1495-1510
    bool pred = false;
    if (chunk < PR && (L >= 32 || lane < L)) {
      const int id = pick<PR>(pi, chunk);
      if (id > 0 && id < np) {
        pred = true;
      } else if (id == 0 && !cz) {
        cz = true;
        pred = true;
      }
    }
    return __ballot_sync(kFull, pred);
  };

  // the list loaded ahead (kAhead) and its node, or -1
  constexpr bool kAhead = !TEAM && !R16 && BR <= 2;
  int ahead_node = -1;
  int ahead[kAhead ? BR : 1];

  // The entry batches and the expansions share one loop, and so one copy of
  // the distance and merge code: a trip gathers a batch's new ids into s_ids,
  // from the entry list while entry batches are left, then from the lists of
  // the nodes it selects.
  // The number of entry batches comes from the parameters alone, so that the
  // branch between the two is uniform to the compiler; a second leaf that
  // equals the first only leaves a batch empty.
  const int max_entries = a.entry_mode == 2                     ? max(L, 2 * a.leaf_cap)
                          : a.entry_mode == 1 && a.max_hits > 1 ? max(L, a.max_hits * a.leaf_cap)
                                                                : L;
  const int n_ebatch = (max_entries + B - 1) / B;
#pragma unroll 1
  for (int eb = 0;;) {
    int n = 0;
    const bool entry = eb < n_ebatch;
    if (entry) {
      // ---- an entry batch (graph_search.cuh:479-959) ----
      // The entry list's bounds are formed here for each batch, so that they
      // hold no registers during the expansions.
      // kd-tree entries from several leaves (mode 1, max_hits H > 1, the
      // reference's multi-hit entry, entry_helper.cu:5-241): every point of
      // each leaf, leaf h in slots [h*cap, (h+1)*cap), -1 leaves as padding,
      // max(L, H*cap) entry slots; the pool keeps the best L.
      const int H = a.entry_mode == 1 ? a.max_hits : 1;
      int hit = a.entry_mode != 0 ? __ldg(a.hits + (size_t)q * H) : 0;
      if (hit < 0 || hit >= a.n_leaves) hit = 0;
      const int32_t* lp = a.leaf_pids + (size_t)hit * a.leaf_cap;
      // learned entries (mode 2): every point of the proposed leaf, then
      // every point of the kd-tree leaf, max(L, both leaves) entry slots in
      // all; the pool keeps the best L of them.  Modes 0 and 1 have L entry
      // slots (:479).
      int hit2 = a.entry_mode == 2 ? __ldg(a.hits2 + q) : -1;
      if (hit2 >= a.n_leaves || hit2 == hit) hit2 = -1;
      const int32_t* lp2 = a.leaf_pids + (size_t)(hit2 < 0 ? 0 : hit2) * a.leaf_cap;
      const int n_first = a.leaf_cap;
      const int n_second = hit2 >= 0 ? a.leaf_cap : 0;
      const int n_entries = a.entry_mode == 2 ? max(L, n_first + n_second)
                            : H > 1            ? max(L, H * a.leaf_cap)
                                               : L;
      // mode 0: the LCGs of reference threads `lane` and `lane + 32`, moved
      // past the earlier batches
      uint32_t seed0 = (uint32_t)q * 64u + (uint32_t)lane;
      uint32_t seed1 = seed0 + 32u;
      auto lcg = [](uint32_t x) { return x * 1103515245u + 12345u; };
      if (a.entry_mode == 0) {
#pragma unroll 1
        for (int i = 0; i < eb * ((BR + 1) / 2); ++i) seed0 = lcg(seed0);
#pragma unroll 1
        for (int i = 0; i < eb * (BR / 2); ++i) seed1 = lcg(seed1);
      }
      const int base = eb * B;
      slots = 0;
#pragma unroll 2
      for (int j = 0; j < BR; ++j) {
        const int slot = (j << 5) + lane;
        const int pos = base + slot;
        int id = np;
        if (slot < B && pos < n_entries) {
          if (a.entry_mode == 0) {
            const uint32_t s = lcg((j & 1) ? seed1 : seed0);
            if (j & 1)
              seed1 = s;
            else
              seed0 = s;
            id = (int)(s % (uint32_t)np);
          } else if (H > 1) {
            const int h = pos / a.leaf_cap, s = pos - h * a.leaf_cap;
            const int lf = h < H ? __ldg(a.hits + (size_t)q * H + h) : -1;
            if (lf >= 0 && lf < a.n_leaves) id = __ldg(a.leaf_pids + (size_t)lf * a.leaf_cap + s);
          } else if (pos < n_first) {
            id = __ldg(lp + pos);
          } else if (hit2 >= 0 && pos < n_first + n_second) {
            id = __ldg(lp2 + pos - n_first);
          }
        }
        bloom.add((uint32_t)id, slot < B && pos < n_entries ? 1u : 0u);  // every entry, padding included (:490)
        n = compact_slot(np, id, j, n, s_ids, slots, lane);
      }
      c_entries += n;
      ++eb;
    } else {
      if (iter >= a.max_iter) break;
      iter++;
      // select up to W unvisited pool slots in pool order; mark them visited
      // by negating the id (:986-1031).  The slots chosen in one register are
      // taken together; the s-th selected node is kept by lane s.
      int my_node = np;
      int nsel = 0;
      const unsigned lt = (1u << lane) - 1u;
      if (BR <= 2 && a.W == 1) {  // the first flagged slot
        if (tmp_flag != 0) {
          const int pos = __ffs(tmp_flag) - 1;
          const int v = __shfl_sync(kFull, pick<PR>(pi, iteration), pos);
          my_node = v < 0 ? -v : v;
#pragma unroll
          for (int j = 0; j < PR; ++j)
            if (j == iteration && lane == pos) pi[j] = -pi[j];
          tmp_flag &= tmp_flag - 1;
          nsel = 1;
        }
      } else
#pragma unroll 1
      while (nsel < a.W && tmp_flag != 0) {
        const int v = pick<PR>(pi, iteration);
        const int rank = __popc(tmp_flag & lt);
        const bool chosen = ((tmp_flag >> lane) & 1u) && rank < a.W - nsel;
        const unsigned took = __ballot_sync(kFull, chosen);
        const int nt = __popc(took);
        if (BR > 2 && a.W == 1) {
          my_node = __shfl_sync(kFull, v, __ffs(took) - 1);
          my_node = my_node < 0 ? -my_node : my_node;
        } else {
          if (chosen) s_ids[nsel + rank] = v < 0 ? -v : v;
          __syncwarp();
          if (lane >= nsel && lane < nsel + nt) my_node = s_ids[lane];
          __syncwarp();
        }
#pragma unroll
        for (int j = 0; j < PR; ++j)
          if (j == iteration && chosen) pi[j] = -pi[j];
        tmp_flag &= ~took;
        nsel += nt;
        if (nsel == a.W) break;
        while (tmp_flag == 0 && iteration < PR) {
          iteration++;
          tmp_flag = scan(iteration);
        }
      }
      if (nsel == 0) break;
      c_expanded += __popc(__ballot_sync(kFull, lane < nsel && my_node < np));
      // The next unvisited pool node, the next iteration's choice unless this
      // one finds a nearer node (it does not in 60 to 80 % of the iterations).
      // One list that fills the batch is loaded ahead, into registers, and
      // used if the choice holds; otherwise the list's lines go to L2 (the
      // reduced-precision paths, which latency bounds; the FP32 path loses
      // more to the prefetches that miss).
      const int next = tmp_flag != 0 ? __shfl_sync(kFull, pick<PR>(pi, iteration), __ffs(tmp_flag) - 1) : -1;
      if (!(kAhead && NR == BR) && PREC != kPrecF32 && next >= 0 && next < np && lane < ((R + 31) >> 5))
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a.graph + (size_t)next * R + 32 * lane));

      // neighbour rows of the selected nodes (:995-1010); a node id >= np
      // expands nothing (the reference would read past the graph)
      if constexpr (R16) {
        // a register holds the lists of two nodes, one per half
        int* s_raw = reinterpret_cast<int*>(s_dist);  // free until the distances
#pragma unroll
        for (int j = 0; j < BR; ++j) {
          const int slot = (j << 5) + lane;
          const int node = __shfl_sync(kFull, my_node, slot >> 4);
          const int id = slot < B && node < np ? __ldg(a.graph + (size_t)node * 16 + (slot & 15)) : np;
          if (slot < B) s_raw[slot] = id;
        }
        // canonical rule: every test of one list sees the filter before any
        // add of that list; lists in selection order.  An id's hashes are
        // computed once for both lists of its register and for test and add:
        // hashed anew for each, 10k queries over 100k BF16 rows of 128 dims,
        // beam 64, took 753 us with one warp each, 651 us now.
        slots = 0;
#pragma unroll 1
        for (int j = 0; 2 * j < nsel; ++j) {
          const int slot = (j << 5) + lane;
          const int id = slot < B ? s_raw[slot] : np;
          uint32_t hb[Bloom::kUnrolled];
          bloom.hash((uint32_t)id, hb);
          bool pass = false;
#pragma unroll
          for (int half = 0; half < (B < 32 ? 1 : 2); ++half) {
            const bool seen = bloom.test(hb) & bloom.test_more((uint32_t)id);
            const bool p = ((lane >> 4) == half) & (id != np) & !seen;
            __syncwarp();
            bloom.add(hb, p ? 1u : 0u);
            bloom.add_more((uint32_t)id, p ? 1u : 0u);
            pass |= p;
            __syncwarp();
          }
          n = compact_slot(np, pass ? id : np, j, n, s_ids, slots, lane);
        }
      } else {
        // canonical rule: every test of one list (NR registers) sees the
        // filter before any add of that list; lists in selection order.
        // Up to KB registers are filtered together, list by list, with their
        // hashes computed ahead.
        constexpr int KB = BR < 4 ? BR : 4;
        slots = 0;
        auto filter = [&](const int (&bi)[KB], int j0) {
          uint32_t hb[KB][Bloom::kUnrolled];
#pragma unroll
          for (int j = 0; j < KB; ++j) bloom.hash((uint32_t)bi[j], hb[j]);
          auto list = [&](auto first, auto count) {
            constexpr int F = decltype(first)::value, N = decltype(count)::value;
            bool pass[N];
#pragma unroll
            for (int j = 0; j < N; ++j) {
              const bool seen = bloom.test(hb[F + j]);
              pass[j] = (bi[F + j] != np) & !seen;
            }
            __syncwarp();
#pragma unroll
            for (int j = 0; j < N; ++j) {
              bloom.add(hb[F + j], pass[j] ? 1u : 0u);
              n = compact_slot(np, pass[j] ? bi[F + j] : np, j0 + F + j, n, s_ids, slots, lane);
            }
            __syncwarp();
          };
          if (NR >= KB) {
            list(Const<0>(), Const<KB>());
          } else if (KB == 4 && NR == 2) {
            list(Const<0>(), Const<KB == 4 ? 2 : 1>());
            list(Const<KB == 4 ? 2 : 0>(), Const<KB == 4 ? 2 : 1>());
          } else {
            list(Const<0>(), Const<1>());
            if constexpr (KB > 1) list(Const<1>(), Const<1>());
            if constexpr (KB > 2) {
              list(Const<2>(), Const<1>());
              list(Const<3>(), Const<1>());
            }
          }
        };
        int bi[BR];
        if (kAhead && NR == BR) {
          if (my_node != ahead_node) {
#pragma unroll
            for (int j = 0; j < BR; ++j) ahead[j] = my_node < np ? __ldg(a.graph + (size_t)my_node * R + (j << 5) + lane) : np;
          }
#pragma unroll
          for (int j = 0; j < BR; ++j) bi[j] = ahead[j];
          ahead_node = next >= 0 && next < np ? next : -1;
          if (ahead_node >= 0) {
#pragma unroll
            for (int j = 0; j < BR; ++j) ahead[j] = __ldg(a.graph + (size_t)next * R + (j << 5) + lane);
          }
        } else {
#pragma unroll
          for (int j = 0; j < BR; ++j) {
            const int s = j >> nr_shift;
            const int node = __shfl_sync(kFull, my_node, s);
            bi[j] = node < np ? __ldg(a.graph + (size_t)node * R + ((j - s * NR) << 5) + lane) : np;
          }
        }
        if (BR <= 4 && bloom.nh <= Bloom::kUnrolled) {
          if constexpr (BR <= 4) filter(bi, 0);
        } else {
          // more registers or hashes: the ids wait in s_dist (free until the
          // distances), where a loop reads them; unrolled over all registers
          // and lists, the filter's code alone outgrew the instruction cache
          int* s_raw = reinterpret_cast<int*>(s_dist);
#pragma unroll
          for (int j = 0; j < BR; ++j) s_raw[(j << 5) + lane] = bi[j];
          if (NR <= KB && bloom.nh <= Bloom::kUnrolled) {
#pragma unroll 1
            for (int j0 = 0; j0 < nsel * NR; j0 += KB) {
              int part[KB];
#pragma unroll
              for (int j = 0; j < KB; ++j) part[j] = s_raw[((j0 + j) << 5) + lane];
              filter(part, j0);
            }
          } else {
#pragma unroll 1
            for (int s = 0; s < nsel; ++s) {
              unsigned pass = 0;
#pragma unroll 1
              for (int r = 0; r < NR; ++r) {
                const int id = s_raw[((s * NR + r) << 5) + lane];
                const bool seen = bloom.test((uint32_t)id);
                if (id != np && !seen) pass |= 1u << r;
              }
              __syncwarp();
#pragma unroll 1
              for (int r = 0; r < NR; ++r) {
                const int j = s * NR + r;
                const int id = s_raw[(j << 5) + lane];
                const uint32_t p = (pass >> r) & 1u;
                bloom.add((uint32_t)id, p);
                n = compact_slot(np, p ? id : np, j, n, s_ids, slots, lane);
              }
              __syncwarp();
            }
          }
        }
      }
      c_dists += n;
    }

    batch_distances<C, NB, PREC, TEAM>(a, qv, qx, s_ids, s_dist, n, lane, t, q, bs);
    // the pool's largest distance: lane 31 of the last register, or lane 15
    // of the 16-slot pool
    const float pmax = __shfl_sync(kFull, pd[PR - 1], NL == 0 ? 15 : 31);
    const int m = __builtin_expect((state & kPoolUnsorted) != 0, 0)
                      ? -1
                      : rank_candidates<NL, NB>(pd, pi, s_ids, s_dist, n, pmax, ties, state, lane);
    merge_batch<NL, NB>(pd, pi, np, s_ids, s_dist, m, slots, ties, lane);
    if (entry) continue;

    bool any = false;
#pragma unroll 1
    for (iteration = 0; iteration < PR; iteration++) {
      tmp_flag = scan(iteration);
      if (tmp_flag != 0) {
        any = true;
        break;
      }
    }
    if ((state & kRebuildAge) == 4) {  // rebuild from the pool (:1518-1529)
      __syncwarp();
      bloom.clear(lane);
      __syncwarp();
#pragma unroll 1
      for (int j = 0; j < PR; ++j) {
        const int v = pick<PR>(pi, j);
        const int id = v < 0 ? -v : v;
        bloom.add((uint32_t)id, id < np ? 1u : 0u);
      }
      __syncwarp();
      state &= ~kRebuildAge;
    }
    ++state;
    if (!any) break;
  }

  // ---- exact FP32 rerank of the final pool (precision paths) ----
  if (PREC != kPrecF32 && a.rerank) {
    // the tensor-core distances read the query from shared memory: its FP32
    // chunks hold no registers until here
    if constexpr (PREC == kPrecBF16 && C >= 1 && C <= 4) load_query_chunks<C>(a, q, lane, qv);
    rerank_pool<C, NL, TEAM>(a, qv, reinterpret_cast<const float*>(q_slot), pd, pi, s_ids, s_dist, lane, t);
  }
  if constexpr (TEAM) {  // releases the helpers
    if (lane == 0) t.ctl[1] = -1;
    team_sync(t);
  }

  // ---- output (:1959-1963) ----
  SearchOut out{a.out_ids, a.out_dists};
  if (a.out_dev) out = *a.out_dev;
#pragma unroll
  for (int j = 0; j < PR; ++j) {
    const int i = (j << 5) + lane;
    if (i < a.k) {
      out.ids[(size_t)q * a.k + i] = pi[j] < 0 ? -pi[j] : pi[j];
      if (out.dists) out.dists[(size_t)q * a.k + i] = pd[j];
    }
  }
  if (a.counters && lane == 0) {
    long long* c = a.counters + (size_t)q * 4;
    c[0] = c_entries;
    c[1] = c_expanded;
    c[2] = c_dists;
    c[3] = iter;
  }
}

// A team member other than the leader, for one query: the query in its own
// registers and slot, then its share of every distance phase the leader
// opens, until the leader ends the query.
template <int C, int PREC>
__device__ __forceinline__ void help_query(const SearchArgs& a, int q, int lane, const int* s_ids,
                                           float* s_dist, uint32_t* q_slot, const Team& t) {
  float qv[qregs(C)];
  QueryExtra<C, PREC> qx;
  load_query<C, PREC>(a, q, lane, qv, qx, q_slot);
  for (;;) {
    team_sync(t);
    const int code = t.ctl[1];
    if (code < 0) break;
    const int n = code & 0xffff;
    if (code >> 16) {  // the exact FP32 rerank of the final pool
      QueryExtra<C, kPrecF32> q32{};
      if constexpr (C == 0) q32.qs = reinterpret_cast<const float*>(q_slot);
      distances<C, kPrecF32, true>(a, qv, q32, s_ids, s_dist, n, lane, t.w, t.K);
    } else {
      distances<C, PREC, true>(a, qv, qx, s_ids, s_dist, n, lane, t.w, t.K);
    }
    team_sync(t);
  }
}

// A warp with no query left: helps the block's searching warps with their
// distance phases until every warp of the block is idle (or, as a safety
// bound, after kHelperIdleLimit scans that found nothing).  A group is taken
// only through the leader's ticket, and only when the ticket's generation
// matches the published (generation, rows) word read after taking it, so a
// stale take of an ended phase is dropped; the leader cannot end a phase
// while a group it counts on is being computed.
template <int C, int NL, int NB, int PREC>
__device__ __noinline__ void help_block(const SearchArgs a, uint32_t* smem, int per_warp, int lane,
                                        BlockShare* bs) {
  constexpr int G = distance_group_size<C, PREC>();
  constexpr int S = batch_slots(NB) > pool_slots(NL) ? batch_slots(NB) : pool_slots(NL);
  const int wpb = blockDim.x >> 5, me = threadIdx.x >> 5;
  if (lane == 0) atomicAdd(&bs->idle, 1u);
  __syncwarp();
  float qv[qregs(C)];
#pragma unroll
  for (int c = 0; c < qregs(C); ++c) qv[c] = 0.0f;
  QueryExtra<C, PREC> qx{};
  long long empty = 0;
  for (;;) {
    if (*reinterpret_cast<volatile unsigned*>(&bs->idle) >= (unsigned)wpb) break;
    bool worked = false;
    for (int w = 0; w < wpb; ++w) {
      if (w == me) continue;
      PhaseDesc& d = bs->desc[w];
      const unsigned long long t0 = *reinterpret_cast<volatile unsigned long long*>(&d.ticket);
      const unsigned long long gn0 = *reinterpret_cast<volatile unsigned long long*>(&d.gen_n);
      if ((t0 >> 32) == 0 || (t0 >> 32) != (gn0 >> 32)) continue;
      if ((int)(unsigned)t0 >= ((int)(unsigned)gn0 + G - 1) / G) continue;
      unsigned long long old = 0;
      if (lane == 0) old = atomicAdd(&d.ticket, 1ull);
      old = __shfl_sync(kFull, old, 0);
      __threadfence_block();
      const unsigned long long gn = *reinterpret_cast<volatile unsigned long long*>(&d.gen_n);
      const unsigned gs = (unsigned)(old >> 32);
      const int grp = (int)(unsigned)old;
      const int n = (int)(unsigned)gn;
      if (gs == 0u || gs != (unsigned)(gn >> 32) || grp >= (n + G - 1) / G) continue;
      const int q = *reinterpret_cast<volatile int*>(&d.q);
      uint32_t* lb = smem + (size_t)w * per_warp;  // the leader's region
      const int* ls_ids = reinterpret_cast<const int*>(lb + a.bloom_words);
      float* ls_dist = reinterpret_cast<float*>(lb + a.bloom_words + S);
      const uint32_t* lslot = lb + a.bloom_words + 2 * S;
      // the leader's query: its shared-memory row, or the FP32 chunks again
      if constexpr (C == 0) {
        qx.qs = reinterpret_cast<const float*>(lslot);
      } else {
        load_query_chunks<C>(a, q, lane, qv);
        if constexpr (PREC == kPrecBF16 && C <= 4) {
          qx.qs = lslot;
          qx.qn = *reinterpret_cast<volatile float*>(&d.qn);
        }
      }
      distance_group<C, PREC>(a, qv, qx, ls_ids, ls_dist, n, lane, grp);
      __syncwarp();
      if (lane == 0) {
        __threadfence_block();
        atomicAdd(&d.done, 1);
      }
      worked = true;
    }
    if (!worked) {
      __nanosleep(256);
      if (++empty > kHelperIdleLimit) break;
    }
  }
}

// Blocks of 8 warps per SM the register budget is set for: 4 (64 registers
// a thread), or 2 (128) for rows of more than 4 chunks in registers and for
// the kernels built for any chunk count with a pool or batch of 8
// registers.  Those spilled over 1 KB at 64 registers; at 128 the 960-d
// search with 256-slot pools and batches ran 1.5x faster on one GB300,
// while the specialised 96- and 128-d kernels of the same pool ran slower.
__host__ __device__ constexpr int search_min_blocks(int C, int NL, int NB) {
  return C > 4 || (C == 0 && (NL >= 8 || NB >= 8)) ? 2 : 4;
}

// The next query of the persistent loop (one lane): the work counter's
// next slot, through the order permutation when there is one (written for
// batches of more than a.order_min queries); nq or more once every query
// is taken.
__device__ __forceinline__ int next_query(const SearchArgs& a, int nq) {
  const int t = (int)atomicAdd(a.work, 1u);
  return a.order && nq > a.order_min && t < nq ? __ldg(a.order + t) : t;
}

template <int C, int NL, int NB, int PREC, bool R16 = false>
__global__ void __launch_bounds__(256, search_min_blocks(C, NL, NB)) search_kernel(SearchArgs a) {
  extern __shared__ uint32_t smem[];
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  constexpr int B = batch_slots(NB);
  constexpr int S = B > pool_slots(NL) ? B : pool_slots(NL);  // compaction slots per warp
  int qwords = kQuerySlotWords;
  if constexpr (C == 0) qwords = query_slot_words_for(0, a.C);
  const int per_warp = a.bloom_words + 2 * S + qwords;
  uint32_t* wbase = smem + (size_t)wib * per_warp;
  Bloom bloom;
  bloom.w = wbase;
  bloom.sw = (uint32_t)__cvta_generic_to_shared(wbase);
  bloom.words_mask = (uint32_t)a.bloom_words - 1u;
  bloom.bits_mask = ((uint32_t)a.bloom_words << 5) - 1u;
  bloom.lw = __ffs(a.bloom_words) - 1;
  bloom.nh = a.bloom_hashes;
  int* s_ids = reinterpret_cast<int*>(wbase + a.bloom_words);
  float* s_dist = reinterpret_cast<float*>(s_ids + S);
  const int nq = a.nq_dev ? *a.nq_dev : a.nq;
  constexpr bool kHelps = tail_helping<C, PREC, NB>();
  BlockShare* bs = nullptr;
  if constexpr (kHelps) {
    bs = block_share(smem, per_warp);
    for (int i = threadIdx.x; i < kBlockShareBytes / 4; i += blockDim.x) reinterpret_cast<uint32_t*>(bs)[i] = 0u;
    __syncthreads();
  }
  for (;;) {
    int q = 0;
    if (lane == 0) q = next_query(a, nq);
    q = __shfl_sync(kFull, q, 0);
    if (q >= nq) break;
    search_query<C, NL, NB, PREC, R16>(a, q, lane, bloom, s_ids, s_dist,
                                       reinterpret_cast<uint32_t*>(s_dist + S), Team(), bs);
  }
  if constexpr (kHelps) help_block<C, NL, NB, PREC>(a, smem, per_warp, lane, bs);
}

// search_kernel with teams of K warps per query (Team): K = a.team, or,
// for a.team < 0, at least a.floor's and otherwise the most (up to 8) that the
// live query count leaves room for in the grid.  K = 1 runs as a team of one.  A kernel of its own, so
// that the single-warp kernel's code and register allocation stay as they
// are; a team never spans blocks (the launch keeps warps per block a
// multiple of K, and K falls back to 1 otherwise).
template <int C, int NL, int NB, int PREC, bool R16 = false>
__global__ void __launch_bounds__(256, search_min_blocks(C, NL, NB)) search_kernel_team(SearchArgs a) {
  extern __shared__ uint32_t smem[];
  dependency_wait();
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  constexpr int B = batch_slots(NB);
  constexpr int S = B > pool_slots(NL) ? B : pool_slots(NL);
  int qwords = kQuerySlotWords;
  if constexpr (C == 0) qwords = query_slot_words_for(0, a.C);
  // per warp: filter, compaction words, query slot, then the team's control
  // words (used in the leader's region)
  const int per_warp = a.bloom_words + 2 * S + qwords + kTeamCtlWords;
  uint32_t* wbase = smem + (size_t)wib * per_warp;
  Bloom bloom;
  bloom.w = wbase;
  bloom.sw = (uint32_t)__cvta_generic_to_shared(wbase);
  bloom.words_mask = (uint32_t)a.bloom_words - 1u;
  bloom.bits_mask = ((uint32_t)a.bloom_words << 5) - 1u;
  bloom.lw = __ffs(a.bloom_words) - 1;
  bloom.nh = a.bloom_hashes;
  const int nq = a.nq_dev ? *a.nq_dev : a.nq;
  const int wpb = blockDim.x >> 5;
  int K = a.team;
  if (K < 0) {  // the floor, then as many as the live batch leaves room for
    const long long total = (long long)gridDim.x * wpb;
    K = a.floor.at(nq, total);
    while (K < 8 && wpb % (2 * K) == 0 && (long long)nq * 2 * K <= total) K *= 2;
  }
  if (K < 1 || K > 8 || wpb % K != 0) K = 1;
  Team t;
  t.K = K;
  t.w = wib & (K - 1);
  t.bar = 1 + wib / K;
  uint32_t* lbase = smem + (size_t)(wib - t.w) * per_warp;  // the leader's region
  t.ctl = reinterpret_cast<volatile int*>(lbase + per_warp - kTeamCtlWords);
  int* ts_ids = reinterpret_cast<int*>(lbase + a.bloom_words);
  float* ts_dist = reinterpret_cast<float*>(ts_ids + S);
  // this warp's own query slot, after its filter and compaction words
  uint32_t* own_slot = wbase + a.bloom_words + 2 * S;
  if (t.w == 0) {
    for (;;) {
      int q = 0;
      if (lane == 0) q = next_query(a, nq);
      q = __shfl_sync(kFull, q, 0);
      if (lane == 0) t.ctl[0] = q;
      team_sync(t);
      if (q >= nq) break;
      search_query<C, NL, NB, PREC, R16, true>(a, q, lane, bloom, ts_ids, ts_dist, own_slot, t);
    }
  } else {
    for (;;) {
      team_sync(t);
      const int q = t.ctl[0];
      if (q >= nq) break;
      help_query<C, PREC>(a, q, lane, ts_ids, ts_dist, own_slot, t);
    }
  }
}

}  // namespace rte
