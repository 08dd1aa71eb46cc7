// fk_sieve.cuh -- the fused sieve kernel (stages S1 and S2).
//
// The line of one item is x = X0 + u*M + R[l]: period u in [0, U), lane l
// over the wheel's admissible residues R mod M.  A CHAIN is one lane over
// Tc 64-period words per thread: either one thread per lane on Tc
// consecutive words, or -- for long lanes -- one warp per lane, thread t
// on words t, t + 32, ... (so a warp's pattern loads are 32 consecutive
// table entries).  32 threads' chains are a BLOCK; the warps of a persistent
// grid claim runs of an item's blocks from the item's counter, so thousands
// of items of uneven length run in one launch.
//
// S1 (pattern sieve).  For the NS pattern primes starting at prime index
// P0 (NS = 24, 32 or 40: a template variant chosen per batch) --
// compile-time constants, so each prime's modulus, word step and
// table offset are immediates -- the kill pattern of 64 consecutive
// periods of a lane is one 64-bit word of a per-prime table of q words,
// indexed by the lane's rotating phase rho (u + s_l) mod q.  The tables
// sit in shared memory, staged from HBM by a bulk async copy (TMA).  This
// is the reference's stage-1a bit-sieve (euler-prime-runs/euler_gpu.py:
// 438-520, dickson-ladders/ladder_gpu.py:254-317, and the AP register
// gather primorial-ap/ap_gpu.py:204-313), re-indexed so that one table per
// prime serves every lane of every wheel.
//
// S2 (compaction rounds).  S1 survivors go through per-thread columns to a
// per-WARP shared-memory queue (no block-wide barrier in the word loop).
// When it fills, the warp drains it: over the first primes one candidate
// per lane, the survivors compacted with ballots between rounds; then one
// prime per lane, every candidate against 32 or 128 primes at once (the
// reference's stage 1b / stage 2 rounds, euler-prime-runs/euler_gpu.py:
// 523-709, dickson-ladders/ladder_gpu.py:349-407, without a host-visible
// queue).  A test is one Montgomery reduction (fk_redc.h) and the engine's
// kill test on the scaled residue.  Final survivors are appended to a
// global candidate list with warp-aggregated atomics.
//
// What bounds it, and what this shape measured (B200, kernel ms): over
// mixed intervals instructions (59% of the issue slots, with 2.5 warps
// waiting for their next one at every issue), in the sparse windows the
// pattern loads' shared-memory wavefronts (50% of the slots, the L1 pipe
// full), two a load.  Against 64-bit Barrett tests with a queue drained at
// every block's end and a CTA barrier after every eight blocks: 256 mixed
// intervals 204 -> 77 ms for the same items (the present choice of sieve
// gives the rounds more of them: 110), the Dickson window of 2^38 j 12.7 ->
// 5.5 with k_rest, the Euler n = 17 windows of 5e14 and 2e16 42.2 -> 23.9 and
// 795 -> 477, the 13# line's quarter 19.3 -> 10.8 with k_rest.
#pragma once
#include "fk_arith.cuh"
#include "fk_types.h"

namespace fk {

constexpr u32 kWaitSpins = 1u << 20;
constexpr u32 kRoundUnroll = 4;  // primes per trip of the compaction rounds

__device__ __forceinline__ u32 smem_u32(const void* p) {
  return (u32)__cvta_generic_to_shared(p);
}

// Entry i of an item's base-residue table: X0 * c1 mod q, the base folded
// into the constants its prime is used with.  A rounds item has one entry
// per prime: the pattern's index up to the first cut, the per-candidate test
// past it.  A marking item has kNSMax entries for the pattern, one per slot
// for the marks and one per prime for the tests past NPm.
__host__ __device__ __forceinline__ u32 mark_tests_at(u32 nslots) {
  return kNSMax + nslots;
}
__device__ __forceinline__ u32 base_entries(const DevEngine& e,
                                            const DevItem& it) {
  return !it.marked ? e.NP
         : mark_tests_at(e.nslots) + (e.NPm < e.NP ? e.NP : 0u);
}
__device__ __forceinline__ u32 base_residue(const DevEngine& e,
                                            const DevItem& it, u32 i) {
  u32 prime = i, c1;
  if (!it.marked) {
    c1 = i < e.rounds[0] ? e.prec[i].c1 : e.trec[i].c1;
  } else if (i < (u32)kNSMax) {
    c1 = e.prec[i].c1;
  } else if (i < mark_tests_at(e.nslots)) {
    prime = e.sprime[i - kNSMax];
    c1 = e.mrec[i - kNSMax].c1;
  } else {
    prime = i - mark_tests_at(e.nslots);
    c1 = e.trec[prime].c1;
  }
  const PrimeRec pr = e.recs[prime];
  const u32 x = fk_bmod128(it.X0_lo, it.X0_hi, pr.q, pr.magic, e.c64[prime]);
  return fk_mulmod(x, c1, pr.q, pr.magic);
}

// ---- per-candidate kill tests ------------------------------------------
// What the tests read besides the prime's record, gathered per item (in
// shared memory for the rounds, from the descriptor for the marking tail).
struct TestCtx {
  const TestRec* trec;
  const ListFilter* filt;
  const u32* kq;        // this item's X0 * c1 mod q
  const u32* lists;
  u32 n, xxmax, xxwords, ap_div;
};

// Dickson: may residue h be on the prime's list (bit 0)?  The three filter
// bits settle nearly every residue off it.
__device__ __forceinline__ u32 list_maybe(const ListFilter& f, u32 h) {
  return ((f.f0 >> (h & 31)) & (f.f1 >> ((h >> 5) & 31)) &
          (f.f2 >> ((h >> 10) & 31))) & 1u;
}
// Is it?  (The list: groups of four, padded with ~0.)
__device__ __forceinline__ bool list_has(const ListFilter& f, u32 h,
                                         const u32* __restrict__ lists) {
  const uint4* l = reinterpret_cast<const uint4*>(lists) + (f.list & 0xFFFFFFu);
  const u32 cnt = f.list >> 24;
  bool k = false;
  for (u32 c = 0; c < cnt; ++c) {
    const uint4 x = __ldg(l + c);
    k |= (x.x == h) | (x.y == h) | (x.z == h) | (x.w == h);
  }
  return k;
}

// Does prime i kill a value of scaled residue r (not Dickson)?  sbits (shared
// memory in the rounds): Euler's bitset of {x^2 + x : x < n}, its last word
// (xxwords) zero.
template <int MODE>
__device__ __forceinline__ bool kill_test(const TestCtx& c, const u32* sbits,
                                          u32 i, const TestRec& t, u32 r) {
  bool kill;
  if (MODE == TEST_AP || MODE == TEST_AP_DIV) {
    kill = r < c.n;
    if (MODE == TEST_AP_DIV && kill && c.filt[i].f0) kill = r == 0;
  } else {
    // r = -x is killed when it is one of the x^2 + x, for the low primes
    // also when r + q, r + 2q, ... is
    kill = (sbits[min(r >> 5, c.xxwords)] >> (r & 31)) & 1u;
    if (MODE == TEST_EULER_LOW)
      for (u32 s = r + t.q; s <= c.xxmax; s += t.q)
        kill |= (sbits[s >> 5] >> (s & 31)) & 1u;
  }
  return kill;
}

// The form an engine's tests take from prime `first` on.
__device__ __forceinline__ u32 test_mode(const DevEngine& e, u32 first) {
  if (e.kind == KIND_DICKSON) return TEST_DICKSON;
  if (e.kind == KIND_AP) return e.ap_div ? TEST_AP_DIV : TEST_AP;
  return first < e.NP && e.trec[first].q > e.xxmax ? TEST_EULER : TEST_EULER_LOW;
}

__device__ __forceinline__ TestRec load_rec(const TestRec* p) {
  const uint4 x = __ldg(reinterpret_cast<const uint4*>(p));
  return TestRec{x.x, x.y, x.z, x.w};
}

__device__ __forceinline__ ListFilter load_filt(const ListFilter* p) {
  const uint4 x = __ldg(reinterpret_cast<const uint4*>(p));
  return ListFilter{x.x, x.y, x.z, x.w};
}

// One prime's data in registers.
template <int MODE>
struct Prime {
  TestRec t;
  ListFilter f;   // Dickson only
  u32 k, i;
  __device__ __forceinline__ void load(const TestCtx& c, u32 p) {
    i = p;
    t = load_rec(c.trec + p);
    k = __ldg(c.kq + p);
    if (MODE == TEST_DICKSON) f = load_filt(c.filt + p);
  }
};

// Does one of the lane's N primes kill the value?  Without a branch, but for
// Dickson's lists, read behind one branch for all N.
template <int MODE, int N>
__device__ __forceinline__ bool any_kill(const Prime<MODE>* p, const TestCtx& c,
                                         const u32* sbits, u32 vl, u32 vh) {
  if (MODE == TEST_DICKSON) {
    u32 h[N], maybe = 0;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const u32 r = redc_residue(p[j].t, p[j].k, vl, vh);
      h[j] = min(r, p[j].t.q - r);
      maybe |= list_maybe(p[j].f, h[j]) << j;
    }
    bool kill = false;
    if (maybe) {
#pragma unroll
      for (int j = 0; j < N; ++j)
        if ((maybe >> j) & 1u) kill |= list_has(p[j].f, h[j], c.lists);
    }
    return kill;
  }
  bool kill = false;
#pragma unroll
  for (int j = 0; j < N; ++j)
    kill |= kill_test<MODE>(c, sbits, p[j].i, p[j].t,
                            redc_residue(p[j].t, p[j].k, vl, vh));
  return kill;
}

// ---- S1 helpers, unrolled over the compile-time pattern primes ----------
// Padding of a variant's pattern tables: entry q + i repeats entry i, so a
// group of G threads on consecutive words reads one run of entries from its
// base index with no wrap inside it.  (With the wrap taken per thread, a
// run that crossed the table's end touched banks twice: 2.45 wavefronts a
// load against 2.)  64 also covers the second word of a step; the variants
// of more primes keep 32 and step twice, to leave room: three CTAs fit an SM
// up to 32 primes (70 to 76 KB each), two at 40 (84 to 92 KB).
template <int NS>
constexpr u32 kPad = NS <= 24 ? kPadWide : kPadNarrow;

// k[I] is the table index of the GROUP's first word for pattern prime I
// (entry k = phase 64k mod q), the same in all its threads: one word forward
// is k + 1 and STRIDE words forward is k + STRIDE (mod q).
template <int P0, int I, int NS>
struct Pat {
  // Two words of the chain, STRIDE words apart, each OR-ed into two
  // accumulators by prime parity, so the loads and ORs of one prime do not
  // wait on the previous prime's; the index then moves 2 * STRIDE words.
  // pt: the tables, advanced by the thread's place in its group.
  template <u32 STRIDE>
  static __device__ __forceinline__ void word2(const u64* __restrict__ pt,
                                               u32* k, u64* acc) {
    constexpr u32 q = fk_nth_prime(P0 + I);
    constexpr u32 off = fk_pat_prefix(P0, I, kPad<NS>);
    constexpr bool once = 2 * STRIDE <= kPad<NS>;
    constexpr u32 st = (once ? 2 * STRIDE : STRIDE) % q;
    const u32 r0 = k[I];
    u32 r1 = r0 + st;
    r1 = min(r1, r1 - q);  // unsigned: r1 - q wraps when r1 < q
    acc[I & 1] |= pt[off + r0];
    if (once) {
      acc[2 + (I & 1)] |= pt[off + r0 + STRIDE];
      k[I] = r1;
    } else {
      acc[2 + (I & 1)] |= pt[off + r1];
      r1 += st;
      k[I] = min(r1, r1 - q);
    }
    Pat<P0, I + 1, NS>::template word2<STRIDE>(pt, k, acc);
  }
};
template <int P0, int NS>
struct Pat<P0, NS, NS> {
  template <u32 STRIDE>
  static __device__ __forceinline__ void word2(const u64*, u32*, u64*) {}
};

// The table indexes of a group of GW threads sweeping lane R from word w0
// (the line offset v = 64 * M * w0 + R): (X0 + v) / (64 * M) mod q, one
// scaled residue each.  Thread t of the group (t) computes the pattern
// primes t, t + GW, ... and the group shares them by shuffle.
template <int NS, int GW>
__device__ __forceinline__ void shared_setup(u32* rho, const TestRec* prec,
                                             const u32* pk, u64 v, u32 t) {
  constexpr int K = (NS + GW - 1) / GW;
  const u32 vl = (u32)v & ((1u << kRedcSplit) - 1u);
  const u32 vh = (u32)(v >> kRedcSplit);
  u32 x[K];
#pragma unroll
  for (int j = 0; j < K; ++j) {
    const u32 i = min(t + (u32)(j * GW), (u32)NS - 1);
    x[j] = redc_residue(prec[i], pk[i], vl, vh);
  }
#pragma unroll
  for (int i = 0; i < NS; ++i)
    rho[i] = GW == 1 ? x[i] : __shfl_sync(0xffffffffu, x[i / GW], i % GW, GW);
}

struct SieveArgs {
  const DevEngine* engines;
  const DevItem* items;
  const u64* task_prefix;  // marking: [nitems + 1] first task of each item
  const u32* item_index;   // [nitems] global item index of each entry
  u32 nitems;
  u32 pad;
  u64 ntask;               // marking: tasks
  const u32* xq;
  u64* cand_key;
  u32* cand_item;
  u64 cand_cap;
  DevCounters* ctr;
  unsigned long long* task_ctr;   // marking: next task
  unsigned long long* block_ctr;  // rounds: [nitems] blocks claimed per item
  // rounds: candidates left in short queues, for k_rest, with the first prime
  // each was not tested against
  u64* rest_key;
  u32* rest_item;
  u32* rest_start;
  u32* rest_state;
  u32 rest_cap;                   // 0: every warp finishes its own
  u32 pad2;
  u32 warp_queue;     // compaction: warp queues below this go one
                      // candidate per warp
  u32 seg_per_task;   // marking: segments per task
};

// Per-warp candidate queues of line offsets v = u * M + R.  A queue
// outlives its warp's blocks and tasks: it is drained when it is full and
// when the CTA moves to another item.  In front of it every thread has a
// column of kColSlots codes (word of the chain << 6 | bit): pushing a
// pattern survivor there takes a store and no vote, and a warp's columns
// are turned into offsets a row at a time, when one is full or the block
// ends.
constexpr u32 kWarps = kBlock / 32;
constexpr u32 kWq = 192;
constexpr u32 kWq2 = 64;
constexpr u32 kColSlots = 16;
constexpr u32 kRestFew = 8;        // fewer candidates than this, with more than
constexpr u32 kRestPrimes = 1024;  // these primes to go, are listed for k_rest

// What a block needs of its item and engine, read from shared memory where
// it is used: held in registers these values would be spilled around the
// calls below, and local memory of 768 threads an SM does not fit in L1.
struct BlockCtx {
  u64 U, M, lo_off, hi_last, nchain;
  const u64* lanes;
  u64 nblock;
  unsigned long long* next;  // the item's counter of claimed blocks
  u32 L, Tc, G, run, gitem;
};

struct SieveSmem {
  u64 queue[kWarps * kWq];
  u64 queue2[kWarps * kWq2];  // past the staged primes
  u64 chain_R[kBlock];    // each thread's chain: its lane and first word
  u64 ntest[kWarps], nword[kWarps];  // work since the last report
  // the first kStaged test primes: every drain starts on these, and a
  // shared load answers in a tenth of the time of one from L2
  TestRec srec[kStaged];
  TestRec prec[kNSMax];   // pattern primes: the scale of their table index
  BlockCtx blk;
  TestCtx ctx;            // the current item's tests
  const u32* rounds;
  u32 entry;              // the item joined
  uint2 sk[kStaged];      // the base's residue; Dickson: the prime's first
                          // word in sbit
  u32 sbit[kStagedBits];  // bit h: min(r, q - r) = h is killed
  u32 chain_w0[kBlock];
  u32 qn[kWarps], qn2[kWarps];  // queue lengths
  u32 pk[kNSMax];
  u32 sbits[kSbits + 1];
  u32 NP, mode, deep;
  u32 eng;
  u32 status;
  unsigned long long mbar;
  unsigned short col[kWarps * kColSlots * 32];
};

// The rounds kernel's shared memory: SieveSmem first, then the pattern
// tables, so a function called out of line finds it at a known shared
// address (through a pointer argument its accesses would be generic loads
// with 64-bit address arithmetic: twice the instructions of a test).
constexpr u32 kSieveSmemBytes = (sizeof(SieveSmem) + 127) / 128 * 128;

__device__ __forceinline__ SieveSmem& sieve_smem_ref() {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  return *reinterpret_cast<SieveSmem*>(smem_raw);
}

// Shared bytes of the first NS pattern primes' tables (the prefix a kernel
// variant stages), padded to 16 bytes.
template <int P0, int NS = kNS, u32 PAD = 0>
__host__ __device__ constexpr u32 pat_bytes() {
  return ((fk_pat_prefix(P0, NS, PAD) + 1) / 2) * 16;
}

// A warp's n candidates against the 32 primes its lanes hold: the survivors
// compacted in place, their count returned.  kills(vl, vh): does the lane's
// prime kill that value?
template <typename F>
__device__ __forceinline__ u32 test_group(u64* Q, u32 n, F kills) {
  const u32 lane = threadIdx.x & 31;
  u32 out = 0;
  for (u32 idx = 0; idx < n; idx += 2) {
    const bool two = idx + 1 < n;
    const u64 v = Q[idx], w = Q[two ? idx + 1 : idx];
    const bool kv = kills((u32)v & ((1u << kRedcSplit) - 1u),
                          (u32)(v >> kRedcSplit));
    const bool kw = kills((u32)w & ((1u << kRedcSplit) - 1u),
                          (u32)(w >> kRedcSplit));
    const bool dv = __any_sync(0xffffffffu, kv);
    const bool dw = __any_sync(0xffffffffu, kw) || !two;
    if (!dv) {
      if (lane == 0) Q[out] = v;  // out <= idx: read already
      ++out;
    }
    if (!dw) {
      if (lane == 0) Q[out] = w;
      ++out;
    }
  }
  __syncwarp();
  return out;
}

// A warp's n candidates against the primes [at, end), 32 at a time, the
// next 32 primes' loads in flight meanwhile.  Returns the survivors' count.
template <int MODE>
__device__ __forceinline__ u32 drain_groups(u64* Q, u32 n, const TestCtx& c,
                                            const u32* sbits, u32 at, u32 end,
                                            u32& ntest) {
  const u32 lane = threadIdx.x & 31;
  if (n == 0 || at >= end) return n;
  Prime<MODE> p, next;
  p.load(c, min(at + lane, end - 1));  // past the end: the last prime again
  for (;;) {
    at += 32;
    next.load(c, min(at + lane, end - 1));
    ntest += n;
    n = test_group(Q, n, [&](u32 vl, u32 vh) {
      return any_kill<MODE, 1>(&p, c, sbits, vl, vh);
    });
    if (at >= end || n == 0) return n;
    p = next;
  }
}

// Append n of the warp's candidates, tested up to prime `at`, to the list
// k_rest finishes, as far as it has room; returns how many it took, from the
// front.  (None when no prime is left: the list holds work, not survivors.)
__device__ __forceinline__ u32 list_rest(const SieveSmem& S, const u64* Q,
                                         u32 n, u32 at, const SieveArgs& a) {
  const u32 lane = threadIdx.x & 31;
  if (n == 0 || a.rest_cap == 0 || at >= S.NP) return 0;
  u64 base = 0;
  if (lane == 0) base = atomicAdd(&a.ctr->nrest, (unsigned long long)n);
  base = __shfl_sync(0xffffffffu, base, 0);
  const u32 m = base < a.rest_cap ? (u32)min((u64)n, a.rest_cap - base) : 0u;
  for (u32 i = lane; i < m; i += 32) {
    a.rest_key[base + i] = Q[i];
    a.rest_item[base + i] = S.blk.gitem;
    a.rest_start[base + i] = at;
    a.rest_state[base + i] = 0;
  }
  return m;
}

// n candidates of a warp's first or second queue, past the first `skip`,
// against every prime from index `at` on, in place, and the survivors into
// the global list: 32 primes at a time, then, once few candidates die among
// 128 primes (S.deep), kDeep groups of 32 at a time (fewer votes, more loads
// in flight).
template <int MODE>
__device__ __noinline__ void drain_rest(bool second, u32 skip, u32 n, u32 at,
                                        const SieveArgs& a) {
  SieveSmem& S = sieve_smem_ref();
  const u32 lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  u64* Q = (second ? S.queue2 + wid * kWq2 : S.queue + wid * kWq) + skip;
  const TestCtx c = S.ctx;
  const u32 NP = S.NP;
  u32 ntest = 0;
  const u32 deep = min(max(S.deep, at), NP);
  n = drain_groups<MODE>(Q, n, c, S.sbits, at, deep, ntest);
  constexpr int kDeep = MODE == TEST_DICKSON ? 2 : 4;
  at = deep;
  bool room = true;
  for (; n > 0 && at + 32 * kDeep <= NP; at += 32 * kDeep) {
    if (room && n < kRestFew && NP - at > kRestPrimes) {
      // too few to be worth this warp's time: k_rest shares them out
      const u32 m = list_rest(S, Q, n, at, a);
      Q += m;
      n -= m;
      room = n == 0;
      if (n == 0) break;
    }
    Prime<MODE> p[kDeep];
#pragma unroll
    for (int j = 0; j < kDeep; ++j) p[j].load(c, at + 32 * j + lane);
    u32 out = 0;
    for (u32 idx = 0; idx < n; ++idx) {
      const u64 v = Q[idx];
      const u32 vl = (u32)v & ((1u << kRedcSplit) - 1u);
      const u32 vh = (u32)(v >> kRedcSplit);
      const bool kill = any_kill<MODE, kDeep>(p, c, S.sbits, vl, vh);
      if (!__any_sync(0xffffffffu, kill)) {
        if (lane == 0) Q[out] = v;  // out <= idx: read already
        ++out;
      }
    }
    ntest += kDeep * n;
    __syncwarp();
    n = out;
  }
  n = drain_groups<MODE>(Q, n, c, S.sbits, at, NP, ntest);
  // survivors: one atomic per warp
  if (n) {
    u64 base = 0;
    if (lane == 0) base = atomicAdd(&a.ctr->ncand, (unsigned long long)n);
    base = __shfl_sync(0xffffffffu, base, 0);
    for (u32 idx = lane; idx < n; idx += 32) {
      if (base + idx < a.cand_cap) {
        a.cand_key[base + idx] = Q[idx];
        a.cand_item[base + idx] = S.blk.gitem;
      } else {
        atomicOr(&a.ctr->overflow, 1u);
      }
    }
  }
  ntest = __reduce_add_sync(0xffffffffu, ntest);
  if (lane == 0) S.ntest[wid] += ntest;
  __syncwarp();
}

// Does a staged prime kill the value?  0 or 1, without a branch.
template <int MODE>
__device__ __forceinline__ u32 staged_kill(const SieveSmem& S, const TestCtx& c,
                                           u32 i, const TestRec& t,
                                           const uint2& k, u32 vl, u32 vh) {
  const u32 r = redc_residue(t, k.x, vl, vh);
  if (MODE == TEST_DICKSON) {
    const u32 h = min(r, t.q - r);
    return (S.sbit[k.y + (h >> 5)] >> (h & 31)) & 1u;
  }
  return kill_test<MODE>(c, S.sbits, i, t, r) ? 1u : 0u;
}

// Drain one warp's queue.  Over the staged primes (the first past the
// pattern, which kill most): rounds with one candidate per lane, the
// survivors compacted in place by ballot after each, down to a.warp_queue
// of them; then one prime per lane.  Those left gather in the warp's
// second queue, until enough of them share the loads of the
// deeper primes' records: there each lane holds one prime and every
// candidate is tested against the warp's 32 primes at once, so no lane
// idles behind a dead candidate.  `final` (the item's end) empties both
// queues, what is left past the staged primes into the list of k_rest while
// that has room.
// Warp-synchronous: every lane calls it.  Not inlined: the pattern loop
// around it keeps its NS table indexes in registers and runs between
// drains.
template <int MODE>
__device__ __noinline__ void warp_drain(bool final, const SieveArgs& a) {
  SieveSmem& S = sieve_smem_ref();
  const u32 wq_short = a.warp_queue;
  const u32 lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const u32 lt = (1u << lane) - 1u;
  u64* Q = S.queue + wid * kWq;
  u64* Q2 = S.queue2 + wid * kWq2;
  u32 n = S.qn[wid], n2 = S.qn2[wid];
  const u32 NP = S.NP, first = __ldg(S.rounds);
  const u32 nstaged = min((u32)kStaged, NP - first);
  if (n > 0) {
    const TestCtx c = S.ctx;
    u32 ntest = 0, at = 0;
    for (u32 r = 0; n >= wq_short && n > 0 && at < nstaged; ++r) {
      // a round's cut, rounded up to whole trips (testing past it is no
      // mistake, and past the last prime the tables repeat it)
      const u32 i0 = at;
      at = min((__ldg(S.rounds + r + 1) - first + kRoundUnroll - 1) /
                   kRoundUnroll * kRoundUnroll, (u32)kStaged);
      u32 out = 0;
      for (u32 base = 0; base < n; base += 32) {
        const u32 idx = base + lane;
        bool alive = idx < n;
        const u64 v = alive ? Q[idx] : 0;
        const u32 vl = (u32)v & ((1u << kRedcSplit) - 1u);
        const u32 vh = (u32)(v >> kRedcSplit);
        // a dead lane idles until the chunk's last candidate dies
        for (u32 i = i0; i < at && __any_sync(0xffffffffu, alive);
             i += kRoundUnroll) {
          if (alive) ntest += kRoundUnroll;
          u32 hit = 0;
#pragma unroll
          for (u32 j = 0; j < kRoundUnroll; ++j) {
            const TestRec t = S.srec[i + j];
            const uint2 k = S.sk[i + j];
            hit |= staged_kill<MODE>(S, c, first + i + j, t, k, vl, vh);
          }
          alive = alive && !hit;
        }
        const u32 bal = __ballot_sync(0xffffffffu, alive);
        if (alive) Q[out + __popc(bal & lt)] = v;  // out <= base: read already
        out += __popc(bal);
      }
      __syncwarp();
      n = out;
    }
    // too few to fill the lanes: one staged prime per lane instead
    for (; n > 0 && at < nstaged; at += 32) {
      const u32 p = min(at + lane, nstaged - 1);
      const TestRec t = S.srec[p];
      const uint2 k = S.sk[p];
      ntest += n;
      n = test_group(Q, n, [&](u32 vl, u32 vh) {
        return staged_kill<MODE>(S, c, first + p, t, k, vl, vh) != 0;
      });
    }
    ntest = __reduce_add_sync(0xffffffffu, ntest);
    if (lane == 0) S.ntest[wid] += ntest;
  }
  const u32 done = first + nstaged;
  if (final) {
    // the warp's last of the item: k_rest shares them out
    u32 m = list_rest(S, Q, n, done, a);
    if (m < n) drain_rest<MODE>(false, m, n - m, done, a);
    m = list_rest(S, Q2, n2, done, a);
    if (m < n2) drain_rest<MODE>(true, m, n2 - m, done, a);
    n = n2 = 0;
  } else if (n >= kWq2 / 2) {   // enough by themselves
    drain_rest<MODE>(false, 0, n, done, a);
    n = 0;
  }
  if (n2 + n > kWq2) {
    drain_rest<MODE>(true, 0, n2, done, a);
    n2 = 0;
  }
  if (lane < n) Q2[n2 + lane] = Q[lane];  // n < kWq2 / 2 = 32
  __syncwarp();
  n2 += n;
  if (lane == 0) {
    S.qn[wid] = 0;
    S.qn2[wid] = n2;
  }
  __syncwarp();
}

static_assert(kWq2 / 2 <= 32, "a lane appends one candidate");

__device__ __forceinline__ void drain_any(SieveSmem& S, bool final,
                                          const SieveArgs& a) {
  if ((S.qn[threadIdx.x >> 5] | S.qn2[threadIdx.x >> 5]) == 0) return;
  switch (S.mode) {
    case TEST_EULER: return warp_drain<TEST_EULER>(final, a);
    case TEST_DICKSON: return warp_drain<TEST_DICKSON>(final, a);
    case TEST_AP: return warp_drain<TEST_AP>(final, a);
    case TEST_EULER_LOW: return warp_drain<TEST_EULER_LOW>(final, a);
    default: return warp_drain<TEST_AP_DIV>(final, a);
  }
}

// Polls the CTA's mbarrier for the given phase, at most `spins` times.
__device__ __forceinline__ bool mbar_wait(u32 mb, u32 phase, u32 spins) {
  u32 done = 0;
  for (u32 i = 0; i < spins && !done; ++i)
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, "
        "[%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(done)
        : "r"(mb), "r"(phase)
        : "memory");
  return done != 0;
}

// Stage the first NS primes' pattern tables of an engine (a prefix of its
// table) into shared memory with one bulk async
// copy (TMA) completing on the CTA's mbarrier, waiting a bounded number of
// polls.  On a timeout it flags the counters (the host reports
// FK_ERR_TIMEOUT) and returns false, after a second bounded wait for the
// copy to land: the CTA then exits, and a copy still writing into the
// shared memory of an exited CTA is what the second wait avoids.  Every
// thread of the CTA calls it.
template <u32 BYTES>
__device__ __forceinline__ bool stage_patterns(u64* spat, const void* pat,
                                               unsigned long long* mbar,
                                               u32* status, u32& phase,
                                               DevCounters* ctr) {
  __syncthreads();
  if (threadIdx.x == 0) {
    *status = 0;
    const u32 mb = smem_u32(mbar);
    const u32 bytes = BYTES;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile(
        "mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb),
        "r"(bytes)
        : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1], %2, [%3];" ::"r"(smem_u32(spat)),
        "l"((u64)__cvta_generic_to_global(pat)), "r"(bytes), "r"(mb)
        : "memory");
    if (!mbar_wait(mb, phase, kWaitSpins)) {
      *status = 1;
      atomicOr(&ctr->overflow, 4u);
      mbar_wait(mb, phase, kWaitSpins);  // let the copy in flight land
    }
  }
  phase ^= 1u;
  __syncthreads();
  return *status == 0;
}

// Move a warp's columns (cn codes in this thread's) into its queue, which
// is drained when a row may not fit.  Not inlined, as warp_drain.
static __device__ __noinline__ void flush_columns(u32 cn, const SieveArgs& a) {
  SieveSmem& S = sieve_smem_ref();
  const u32 wl = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned short* C = S.col + wid * (kColSlots * 32) + wl;
  const u32 rows = __reduce_max_sync(0xffffffffu, cn);
  // the queue's length, the same in every lane; lane 0 stores it only after
  // all have read it, for the drain and for the next flush
  u32 qn = S.qn[wid];
  __syncwarp();
  for (u32 r = 0; r < rows; ++r) {
    const u32 bal = __ballot_sync(0xffffffffu, r < cn);
    if (qn + 32 > kWq) {
      if (wl == 0) S.qn[wid] = qn;
      __syncwarp();   // and the entries pushed so far are in the queue
      drain_any(S, false, a);
      qn = 0;
    }
    if (r < cn) {
      const u32 code = C[32 * r];
      const u64 u = 64ull * (S.chain_w0[threadIdx.x] + (code >> 6) * S.blk.G) +
                    (code & 63u);
      S.queue[wid * kWq + qn + __popc(bal & ((1u << wl) - 1u))] =
          u * S.blk.M + S.chain_R[threadIdx.x];
    }
    qn += __popc(bal);
  }
  if (wl == 0) S.qn[wid] = qn;
  __syncwarp();
}

// Push the set bits of one 32-bit half word into the thread's column while
// it has room; the bits pushed are cleared.
__device__ __forceinline__ void push_half(u32& x, u32 code, unsigned short* C,
                                          u32& cn) {
  while (x != 0 && cn < kColSlots) {
    const u32 b = 31u - __clz((int)x);
    x ^= 1u << b;
    C[32 * cn] = (unsigned short)(code + b);
    ++cn;
  }
}

// The periods of word w the item covers, of which R's are admitted: all 64
// except in the item's first word (lo_off) and its last (U, hi_last).
__device__ __forceinline__ u64 word_mask(const BlockCtx& c, u32 w, u64 R) {
  if (64ull * w >= c.U) return 0;
  const u64 left = c.U - 64ull * w;
  u64 m = left >= 64 ? ~0ull : (1ull << left) - 1ull;
  if (w == 0 && R < c.lo_off) m &= ~1ull;
  if (left <= 64 && R >= c.hi_last) m &= ~(1ull << (left - 1));
  return m;
}

// One block of 32 threads' chains: thread wl of the warp sweeps chain
// g = gw + (wl >> log2 G) of the item and pushes its pattern survivors
// through its column into the warp's queue.
template <int P0, int NS>
__device__ __forceinline__ void sieve_block(const u64* __restrict__ spat,
                                            SieveSmem& S, const SieveArgs& a,
                                            u64 gw) {
  const u32 wl = threadIdx.x & 31, wid = threadIdx.x >> 5;
  u32 G = S.blk.G, Tc = S.blk.Tc;
  // words of this thread's chain inside the item, and the fewest over the
  // warp: words 1 ... least - 2 of every chain are whole
  u32 words = 0;
  u32 rho[NS];
  {
    const u32 gsh = G == 32 ? 5u : (G == 8 ? 3u : 0u);
    const u32 L = S.blk.L;
    const u64 nchain = S.blk.nchain, g = gw + (wl >> gsh);
    u32 chunk = 0, lane = 0;   // chunks per lane: below 2^30 words
    const bool active = g < nchain;
    if (active) {
      if (nchain <= 0xFFFFFFFFull) {
        chunk = (u32)g / L;
        lane = (u32)g - chunk * L;
      } else {
        chunk = (u32)(g / L);
        lane = (u32)(g % L);
      }
    }
    const u64 R = active ? S.blk.lanes[lane] : 0;
    const u32 w0 = chunk * (G * Tc) + (wl & (G - 1));
    const u32 wend = (u32)((S.blk.U + 63) >> 6);
    if (active && w0 < wend) words = min(Tc, (wend - w0 + G - 1) / G);
    S.chain_R[threadIdx.x] = R;
    S.chain_w0[threadIdx.x] = w0;
    // the group's first word is chunk * G * Tc
    const u64 v0 = 64ull * S.blk.M * (chunk * (G * Tc)) + R;
    if (G == 32)
      shared_setup<NS, 32>(rho, S.prec, S.pk, v0, wl);
    else if (G == 8)
      shared_setup<NS, 8>(rho, S.prec, S.pk, v0, wl & 7u);
    else
      shared_setup<NS, 1>(rho, S.prec, S.pk, v0, 0);
  }
  const u32 total = __reduce_add_sync(0xffffffffu, words);
  u32 least = __reduce_min_sync(0xffffffffu, words);
  if (wl == 0) S.nword[wid] += total;
  const u64* pt = spat + (wl & (G - 1));
  unsigned short* C = S.col + wid * (kColSlots * 32) + wl;
  u32 cn = 0;
  for (u32 wi = 0; wi < Tc; wi += 2) {
    // two words of the chain: j = wi and wi + 1
    u64 acc[4] = {0, 0, 0, 0};
    if (G == 32)
      Pat<P0, 0, NS>::template word2<32>(pt, rho, acc);
    else if (G == 8)
      Pat<P0, 0, NS>::template word2<8>(pt, rho, acc);
    else
      Pat<P0, 0, NS>::template word2<1>(pt, rho, acc);
    u64 s0 = ~(acc[0] | acc[1]), s1 = ~(acc[2] | acc[3]);
    if (wi == 0 || wi + 2 >= least) {
      const u64 R = S.chain_R[threadIdx.x];
      const u32 w = S.chain_w0[threadIdx.x] + wi * G;
      s0 = wi < words ? s0 & word_mask(S.blk, w, R) : 0ull;
      s1 = wi + 1 < words ? s1 & word_mask(S.blk, w + G, R) : 0ull;
    }
    // into the columns; a full one empties the warp's
    u32 x[4] = {(u32)s0, (u32)(s0 >> 32), (u32)s1, (u32)(s1 >> 32)};
    for (;;) {
#pragma unroll
      for (int k = 0; k < 4; ++k) push_half(x[k], (wi << 6) + 32 * k, C, cn);
      if (!__any_sync(0xffffffffu, (x[0] | x[1] | x[2] | x[3]) != 0)) break;
      // the loop's values wait out the flush in local memory: live across
      // the call they would be spilled in the word loop instead
      volatile u32 keep[NS + 9];
#pragma unroll
      for (int i = 0; i < NS; ++i) keep[i] = rho[i];
#pragma unroll
      for (int k = 0; k < 4; ++k) keep[NS + k] = x[k];
      keep[NS + 4] = wi;
      keep[NS + 5] = words;
      keep[NS + 6] = least;
      keep[NS + 7] = Tc;
      keep[NS + 8] = G;
      flush_columns(cn, a);
      cn = 0;
#pragma unroll
      for (int i = 0; i < NS; ++i) rho[i] = keep[i];
#pragma unroll
      for (int k = 0; k < 4; ++k) x[k] = keep[NS + k];
      wi = keep[NS + 4];
      words = keep[NS + 5];
      least = keep[NS + 6];
      Tc = keep[NS + 7];
      G = keep[NS + 8];
    }
  }
  // the codes refer to this block's chains
  flush_columns(cn, a);
}

// The first entry of the family's list with blocks left, from `from` on
// and around; nitems when none has.  Called by one whole warp.
__device__ __forceinline__ u32 find_item(const SieveArgs& a, u32 from) {
  const u32 wl = threadIdx.x & 31;
  for (u32 k = 0; k < a.nitems; k += 32) {
    u32 e = from + k + wl;
    if (e >= a.nitems) e -= a.nitems;
    const bool left = k + wl < a.nitems &&
                      *(volatile unsigned long long*)(a.block_ctr + e) <
                          a.items[a.item_index[e]].ntask;
    const u32 bal = __ballot_sync(0xffffffffu, left);
    if (bal) return __shfl_sync(0xffffffffu, e, __ffs((int)bal) - 1);
  }
  return a.nitems;
}

// Where in the list a CTA starts: by its SM, the SM's CTAs side by side.  The
// list is sorted by kind of test, so an SM's CTAs run the same code most of
// the time: with the kinds mixed on every SM 2.85 warps waited for
// instructions at every issue, now 2.30 (1.98 with the AP items alone), and
// the rounds of 256 mixed intervals took 112.6 ms, now 108.1.
__device__ __forceinline__ u32 first_item(u32 nitems) {
  u32 sm, nsm;
  asm("mov.u32 %0, %%smid;" : "=r"(sm));
  asm("mov.u32 %0, %%nsmid;" : "=r"(nsm));
  const u32 per = (gridDim.x + nsm - 1) / nsm;
  const u64 at = (u64)sm * per + blockIdx.x / nsm;
  return (u32)min(at * nitems / ((u64)nsm * per), (u64)nitems - 1);
}

// NS: the pattern primes this variant stages (the engine descriptor's NS
// and round cuts must match it).  A CTA joins an item -- stages its
// engine's tables and its base residues -- and its warps claim runs of the
// item's blocks from the item's counter until none is left, each at its own
// pace; then they drain their queues and the CTA joins the next item with
// work.  The SMs start spread over the list, so short items run side by side
// and long ones draw every CTA in the end.  The variants of 40 primes, of
// which two CTAs fit an SM, take the registers of two: 128 mixed intervals of
// up to 2^33, all in the rounds, 137.8 -> 126.5 ms.  (With CTA-wide tasks the
// barrier ending each one cost a fifth to a third of the warps' time: a
// warp in a drain held up the other seven.)
template <int P0, int NS>
__global__ void __launch_bounds__(kBlock, NS <= 32 ? 3 : 2)
    k_sieve(const __grid_constant__ SieveArgs a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  SieveSmem& S = sieve_smem_ref();
  u64* spat = reinterpret_cast<u64*>(smem_raw + kSieveSmemBytes);
  const u32 tid = threadIdx.x, wl = tid & 31, wid = tid >> 5;
  if (tid == 0) {
    S.eng = 0xFFFFFFFFu;
    const u32 mb = smem_u32(&S.mbar);
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb)
                 : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (wl == 0) {
    S.qn[wid] = S.qn2[wid] = 0;
    S.ntest[wid] = S.nword[wid] = 0;
  }
  u32 phase = 0;
  u32 entry = first_item(a.nitems);
  for (;;) {
    if (wid == 0) {
      const u32 e = find_item(a, entry);
      if (wl == 0) S.entry = e;
    }
    __syncthreads();   // and every warp is past the old item's tables
    entry = S.entry;
    if (entry >= a.nitems) break;
    {
      const u32 gitem = a.item_index[entry];
      const DevItem& it = a.items[gitem];
      const u32 eidx = it.engine;
      const DevEngine& eg = a.engines[eidx];
      if (S.eng != eidx) {
        // ---- engine switch: stage its pattern table into shared memory ----
        if (!stage_patterns<pat_bytes<P0, NS, kPad<NS>>()>(
                spat, kPad<NS> == kPadWide ? eg.patw : eg.patn, &S.mbar,
                &S.status, phase, a.ctr))
          return;
        if (tid < (u32)NS) S.prec[tid] = eg.prec[tid];
        for (u32 i = tid; i <= eg.sbits_words; i += kBlock)
          S.sbits[i] = i < eg.sbits_words ? eg.sbits[i] : 0u;
        __syncthreads();   // and every warp has read S.eng
        if (tid == 0) S.eng = eidx;
      }
      if (tid < (u32)NS) S.pk[tid] = a.xq[it.xq_off + tid];
      const u32 first = eg.rounds[0];
      if (tid < (u32)kStaged && first < eg.NP) {
        const u32 p = min(first + tid, eg.NP - 1);  // past the end: the last
        S.srec[tid] = eg.trec[p];
        S.sk[tid] = make_uint2(
            a.xq[it.xq_off + p],
            eg.kind == KIND_DICKSON
                ? eg.boff[p - kNSMin] - eg.boff[first - kNSMin] : 0u);
      }
      if (eg.kind == KIND_DICKSON && first < eg.NP) {
        const u32 b0 = eg.boff[first - kNSMin];
        const u32 b1 = eg.boff[min(first + kStaged, eg.NP) - kNSMin];
        for (u32 i = b0 + tid; i < b1; i += kBlock) S.sbit[i - b0] = eg.bits[i];
      }
      if (tid == 0) {
        S.ctx = TestCtx{eg.trec, eg.filt, a.xq + it.xq_off, eg.lists,
                        eg.n, eg.xxmax, eg.sbits_words, eg.ap_div};
        S.blk = BlockCtx{it.U, eg.M, it.lo_off, it.hi_last, it.nchunk * eg.L,
                         reinterpret_cast<const u64*>(eg.lanes), it.ntask,
                         a.block_ctr + entry, eg.L, it.Tc, it.lane_threads,
                         it.run, gitem};
        S.rounds = eg.rounds;
        S.NP = eg.NP;
        S.deep = eg.deep;
        S.mode = test_mode(eg, first);
      }
      __syncthreads();
    }
    for (;;) {
      u64 b = 0;
      if (wl == 0) b = atomicAdd(S.blk.next, (unsigned long long)S.blk.run);
      b = __shfl_sync(0xffffffffu, b, 0);
      if (b >= S.blk.nblock) break;
      const u64 end = min(b + S.blk.run, S.blk.nblock);
      for (; b < end; ++b) {
        const u32 G = S.blk.G;
        // chains per block: 32 / G
        sieve_block<P0, NS>(spat, S, a,
                            b * (G == 32 ? 1u : (G == 8 ? 4u : 32u)));
      }
    }
    // drain the queues and report
    drain_any(S, true, a);
    if (wl == 0) {
      if (S.ntest[wid]) atomicAdd(&a.ctr->s2_tests, S.ntest[wid]);
      if (S.nword[wid]) atomicAdd(&a.ctr->s1_words, S.nword[wid]);
      S.ntest[wid] = S.nword[wid] = 0;
    }
    __syncwarp();
    if (++entry == a.nitems) entry = 0;
  }
}

}  // namespace fk
