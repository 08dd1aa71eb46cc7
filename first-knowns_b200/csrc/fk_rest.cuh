// fk_rest.cuh -- the candidates the rounds kernel's warps were left with.
//
// A warp that reaches its item's end, or whose queue has come down to a few
// candidates, holds candidates with thousands of primes before them: alone
// they cost it a chain of dependent loads (milliseconds with 82,000 primes),
// while the warps beside it are done.  They come here instead, listed, and are
// shared out: eight neighbours of the list against one chunk of the primes
// are a unit, the first chunks of all before the second ones, so a later
// chunk mostly finds its candidates dead already.  The warp that finishes a
// candidate's last chunk emits it.
#pragma once
#include "fk_sieve.cuh"

namespace fk {

constexpr u32 kRestChunk = 512;       // primes per unit
constexpr u32 kRestGroup = 8;         // candidates per unit: they share the
                                      // loads of the primes' records, which
                                      // one by one would be bound by L2
constexpr u32 kRestDead = 0x80000000u;

// The candidates `alive` (bits; lane i holds candidate i's offset v) against
// the primes [at, end): those no prime kills.
template <int MODE>
__device__ __forceinline__ u32 rest_group(const TestCtx& c, const u32* sbits,
                                          u64 v, u32 alive, u32 at, u32 end,
                                          u32& ntest) {
  const u32 lane = threadIdx.x & 31;
  const u32 vl = (u32)v & ((1u << kRedcSplit) - 1u);
  const u32 vh = (u32)(v >> kRedcSplit);
  constexpr int kDeep = 4;
  for (; at < end && alive; at += 32 * kDeep) {
    Prime<MODE> p[kDeep];
#pragma unroll
    for (int j = 0; j < kDeep; ++j)   // past the end: the last prime again
      p[j].load(c, min(at + 32 * j + lane, end - 1));
    for (u32 m = alive; m; m &= m - 1) {
      const u32 i = __ffs((int)m) - 1;
      const u32 l = __shfl_sync(0xffffffffu, vl, i);
      const u32 h = __shfl_sync(0xffffffffu, vh, i);
      const bool kill = any_kill<MODE, kDeep>(p, c, sbits, l, h);
      ntest += kDeep;
      if (__any_sync(0xffffffffu, kill)) alive &= ~(1u << i);
    }
  }
  return alive;
}

// max_np: the most sieve primes of the batch's engines.
__global__ void __launch_bounds__(kBlock)
    k_rest(const __grid_constant__ SieveArgs a, u32 max_np) {
  const u32 n = (u32)min((u64)a.ctr->nrest, (u64)a.rest_cap);
  const u32 lane = threadIdx.x & 31;
  const u32 warps = gridDim.x * (kBlock / 32);
  const u32 groups = (n + kRestGroup - 1) / kRestGroup;
  const u64 units = (u64)groups * ((max_np + kRestChunk - 1) / kRestChunk);
  u32 ntest = 0;
  for (u64 u = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; u < units;
       u += warps) {
    const u32 k = (u32)(u / groups), at = k * kRestChunk;
    const u32 i = (u32)(u % groups) * kRestGroup + lane;
    const bool mine = lane < kRestGroup && i < n;
    const u32 item = mine ? a.rest_item[i] : 0u;
    const u64 v = mine ? a.rest_key[i] : 0ull;
    const u32 start = mine ? a.rest_start[i] : 0u;
    const u32 np = mine ? a.engines[a.items[item].engine].NP : 0u;
    // this chunk has primes the candidate was not tested against
    bool todo = mine && at < np && min(at + kRestChunk, np) > start &&
                !(*(volatile u32*)(a.rest_state + i) & kRestDead);
    for (u32 left; (left = __ballot_sync(0xffffffffu, todo)) != 0;) {
      // those of one item together
      const u32 it0 = __shfl_sync(0xffffffffu, item, __ffs((int)left) - 1);
      const u32 mask = __ballot_sync(0xffffffffu, todo && item == it0);
      const DevItem& it = a.items[it0];
      const DevEngine& e = a.engines[it.engine];
      const u32 end = min(at + kRestChunk, e.NP);
      // from the earliest start among them, in whole groups of 32
      u32 from = __reduce_min_sync(0xffffffffu,
                                   todo && item == it0 ? start : 0xFFFFFFFFu);
      from = max(from, at);
      const TestCtx c{e.trec, e.filt, a.xq + it.xq_off, e.lists,
                      e.n, e.xxmax, e.sbits_words, e.ap_div};
      u32 alive;
      switch (test_mode(e, e.rounds[0])) {
        case TEST_EULER:
          alive = rest_group<TEST_EULER>(c, e.sbits, v, mask, from, end, ntest);
          break;
        case TEST_DICKSON:
          alive = rest_group<TEST_DICKSON>(c, e.sbits, v, mask, from, end, ntest);
          break;
        case TEST_AP:
          alive = rest_group<TEST_AP>(c, e.sbits, v, mask, from, end, ntest);
          break;
        case TEST_EULER_LOW:
          alive = rest_group<TEST_EULER_LOW>(c, e.sbits, v, mask, from, end, ntest);
          break;
        default:
          alive = rest_group<TEST_AP_DIV>(c, e.sbits, v, mask, from, end, ntest);
          break;
      }
      if (todo && item == it0) {
        todo = false;
        const u32 chunks = (np + kRestChunk - 1) / kRestChunk - start / kRestChunk;
        if (!((alive >> lane) & 1u)) {
          atomicOr(a.rest_state + i, kRestDead);
        } else if ((atomicAdd(a.rest_state + i, 1u) & ~kRestDead) + 1 == chunks) {
          // every chunk is done and none killed it (one that does, or finds
          // it dead, never counts)
          const u64 p = atomicAdd(&a.ctr->ncand, 1ull);
          if (p < a.cand_cap) {
            a.cand_key[p] = v;
            a.cand_item[p] = item;
          } else {
            atomicOr(&a.ctr->overflow, 1u);
          }
        }
      }
    }
  }
  ntest = __reduce_add_sync(0xffffffffu, ntest);
  if (lane == 0 && ntest) atomicAdd(&a.ctr->s2_tests, (unsigned long long)ntest);
}

}  // namespace fk
