// fk_sieve.cuh -- the fused sieve kernel (stages S1 and S2).
//
// The line of one item is x = X0 + u*M + R[l]: period u in [0, U), lane l
// over the wheel's admissible residues R mod M.  A CHAIN is one lane over
// Tc 64-period words per thread: either one thread per lane on Tc
// consecutive words, or -- for long lanes -- one warp per lane, thread t
// on words t, t + 32, ... (so a warp's pattern loads are 32 consecutive
// table entries).  32 threads' chains are a BLOCK; a CTA task is a run of
// one item's blocks, pulled from a device counter by a persistent grid, so
// thousands of items of uneven length run in one launch, and inside a task
// the warps claim blocks from a shared counter.
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
// What bounds it, and what this shape measured (B200, kernel ms against
// the 64-bit Barrett tests with a queue drained at every block's end): the
// kernel issues instructions, so the tests' length is what counts -- 10
// to 20 warp instructions a test against 58 -- then the pattern loads'
// shared-memory wavefronts.  256 mixed intervals 204 -> 119 ms, the Dickson
// window of 2^38 j 12.7 -> 7.8, the Euler n = 17 windows of 5e14 and 2e16
// 42.2 -> 32.2 and 795 -> 627, the 13# line's quarter 19.3 -> 15.5.
#pragma once
#include "fk_arith.cuh"
#include "fk_types.h"

namespace fk {

constexpr u32 kWaitSpins = 1u << 20;
constexpr u32 kRoundUnroll = 4;  // primes per trip of the compaction rounds

__device__ __forceinline__ u32 smem_u32(const void* p) {
  return (u32)__cvta_generic_to_shared(p);
}

// Block-wide exclusive scan of one u32 per thread; returns the prefix and
// sets *total.  Two barriers.
__device__ __forceinline__ u32 block_scan(u32 v, u32* s_warp, u32* total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  u32 x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    u32 y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[wid] = x;
  __syncthreads();
  u32 base = 0, tot = 0;
#pragma unroll
  for (int w = 0; w < kBlock / 32; ++w) {
    u32 t = s_warp[w];
    base += (w < wid) ? t : 0;
    tot += t;
  }
  __syncthreads();
  *total = tot;
  return base + x - v;
}

// The base of every (item, prime) of sieve items: X0 mod q for the primes
// sieved by pattern or mark, X0 * c1 mod q for those tested per candidate
// (the rounds' from their first cut, the marking sieve's past NPm).
__device__ __forceinline__ u32 base_residue(const DevEngine& e,
                                            const DevItem& it, u32 i) {
  const PrimeRec pr = e.recs[i];
  const u32 x = fk_bmod128(it.X0_lo, it.X0_hi, pr.q, pr.magic, e.c64[i]);
  const u32 first = it.marked ? e.NPm : e.rounds[0];
  return i < first ? x : fk_mulmod(x, e.trec[i].c1, pr.q, pr.magic);
}

// ---- per-candidate kill tests ------------------------------------------
// What the tests read besides the prime's record, gathered per item (in
// shared memory for the rounds, from the descriptor for the marking tail).
struct TestCtx {
  const TestRec* trec;
  const ListFilter* filt;
  const u32* kq;        // this item's X0 * c1 mod q
  const u32* lists;
  const u32* sbits;     // Euler: bitset of {x^2 + x : x < n}
  u32 n, xxmax, xxwords, ap_div;
};

// Is residue r on the prime's list?  The three filter bits settle nearly
// every residue off it; the list itself (groups of four, padded with ~0) is
// read only behind them.
__device__ __forceinline__ bool list_kill(const ListFilter& f, u32 r,
                                          const u32* __restrict__ lists) {
  if (!((f.f0 >> (r & 31)) & (f.f1 >> ((r >> 5) & 31)) &
        (f.f2 >> ((r >> 10) & 31)) & 1u))
    return false;
  const uint4* l = reinterpret_cast<const uint4*>(lists) + (f.list & 0xFFFFFFu);
  const u32 cnt = f.list >> 24;
  bool k = false;
  for (u32 c = 0; c < cnt; ++c) {
    const uint4 x = __ldg(l + c);
    k |= (x.x == r) | (x.y == r) | (x.z == r) | (x.w == r);
  }
  return k;
}

// Does prime i kill a value of scaled residue r (Euler, AP)?
template <int KIND>
__device__ __forceinline__ bool kill_test(const TestCtx& c, u32 i,
                                          const TestRec& t, u32 r) {
  bool kill;
  if (KIND == KIND_AP) {
    kill = r < c.n;
    if (c.ap_div && kill && c.filt[i].f0) kill = r == 0;
  } else {
    // r = -x is killed when it is one of the x^2 + x: the bitset's last
    // word (xxwords) is zero
    kill = (c.sbits[min(r >> 5, c.xxwords)] >> (r & 31)) & 1u;
    // the primes up to max(x^2 + x): so are r + q, r + 2q, ...
    if (t.q <= c.xxmax)
      for (u32 s = r + t.q; s <= c.xxmax; s += t.q)
        kill |= (c.sbits[s >> 5] >> (s & 31)) & 1u;
  }
  return kill;
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
template <int KIND>
struct Prime {
  TestRec t;
  ListFilter f;   // Dickson only
  u32 k, i;
  __device__ __forceinline__ void load(const TestCtx& c, u32 p) {
    i = p;
    t = load_rec(c.trec + p);
    k = __ldg(c.kq + p);
    if (KIND == KIND_DICKSON) f = load_filt(c.filt + p);
  }
  __device__ __forceinline__ bool kills(const TestCtx& c, u32 vl,
                                        u32 vh) const {
    const u32 r = redc_residue(t, k, vl, vh);
    if (KIND == KIND_DICKSON) return list_kill(f, min(r, t.q - r), c.lists);
    return kill_test<KIND>(c, i, t, r);
  }
};

// ---- S1 helpers, unrolled over the compile-time pattern primes ----------
// k[I] is the lane's current TABLE INDEX for pattern prime I (entry k =
// phase 64k mod q), so one word forward is k + 1 and STRIDE words forward
// is k + STRIDE (mod q).
template <int P0, int I, int NS>
struct Pat {
  // Two words of the chain, STRIDE words apart, each OR-ed into two
  // accumulators by prime parity, so the loads and ORs of one prime do not
  // wait on the previous prime's; the index then moves 2 * STRIDE words.
  template <u32 STRIDE>
  static __device__ __forceinline__ void word2(const u64* __restrict__ spat,
                                               u32* k, u64* acc) {
    constexpr u32 q = fk_nth_prime(P0 + I);
    constexpr u32 off = fk_pat_prefix(P0, I);
    constexpr u32 st = STRIDE % q;
    const u32 r0 = k[I];
    u32 r1 = r0 + st;
    r1 = min(r1, r1 - q);  // unsigned: r1 - q wraps when r1 < q
    u32 r2 = r1 + st;
    r2 = min(r2, r2 - q);
    acc[I & 1] |= spat[off + r0];
    acc[2 + (I & 1)] |= spat[off + r1];
    k[I] = r2;
    Pat<P0, I + 1, NS>::template word2<STRIDE>(spat, k, acc);
  }
  // The table index of period u0 of lane R: phase (u0 + s_l) mod q with
  // s_l = (X0 + R) * (M mod q)^-1, times 64^-1 (s_minv already carries it).
  static __device__ __forceinline__ void setup(u32* k, u64 R, u64 u0,
                                               const u32* __restrict__ xq,
                                               const u32* s_minv) {
    constexpr u32 q = fk_nth_prime(P0 + I);
    constexpr u32 i64 = fk_inv64(q);
    const u32 rq = (u32)(R % q);
    const u32 s = (u32)(((xq[I] + rq) % q) * (u64)s_minv[I] % q);
    k[I] = (u32)(((u32)(u0 % q) * i64 + s) % q);
    Pat<P0, I + 1, NS>::setup(k, R, u0, xq, s_minv);
  }
  // The table indexes of a group of GW threads sweeping one lane, thread
  // t of the group from word base + t: (base_I + t) mod q, base_I held in
  // v[I / GW] by thread I mod GW of the group.
  template <int GW>
  static __device__ __forceinline__ void spread(u32* k, const u32* v,
                                                u32 t) {
    constexpr u32 q = fk_nth_prime(P0 + I);
    const u32 b = __shfl_sync(0xffffffffu, v[I / GW], I % GW, GW);
    // t < GW: below q for every prime when GW = 8 and from the 37 up when
    // GW = 32; the 17 ... 31 of the 13# and 17# families reduce it first,
    // so one subtraction still ends in [0, q)
    const u32 r = b + (q >= (u32)GW ? t : t % q);
    k[I] = min(r, r - q);
    Pat<P0, I + 1, NS>::template spread<GW>(k, v, t);
  }
};
template <int P0, int NS>
struct Pat<P0, NS, NS> {
  template <u32 STRIDE>
  static __device__ __forceinline__ void word2(const u64*, u32*, u64*) {}
  static __device__ __forceinline__ void setup(u32*, u64, u64, const u32*,
                                               const u32*) {}
  template <int GW>
  static __device__ __forceinline__ void spread(u32*, const u32*, u32) {}
};

// Pattern prime I's table index at word wb of lane R: (wb + s) mod q with
// s = (X0 + R) * (M mod q)^-1 * 64^-1 mod q the lane's phase (xq holds X0
// mod q, s_minv the product of the two inverses), from the prime's record.
__device__ __forceinline__ u32 lane_base(const DevEngine& e,
                                         const u32* __restrict__ xq,
                                         const u32* s_minv, u64 R, u64 wb,
                                         u32 I) {
  const PrimeRec pr = e.recs[I];
  u32 x = xq[I] + fk_bmod(R, pr.q, pr.magic);
  x = min(x, x - pr.q);
  const u32 s = fk_mulmod(x, s_minv[I], pr.q, pr.magic);
  const u32 t = s + fk_bmod(wb, pr.q, pr.magic);
  return min(t, t - pr.q);
}

// The table indexes of a group of GW threads sweeping one lane from word
// wb, thread t at word wb + t: thread t computes the base index of the
// pattern primes t, t + GW, ... and the group shares them by shuffle.
template <int P0, int NS, int GW>
__device__ __forceinline__ void shared_setup(u32* rho, const DevEngine& e,
                                             const u32* __restrict__ xq,
                                             const u32* s_minv, u64 R,
                                             u64 wb, u32 t) {
  constexpr int K = (NS + GW - 1) / GW;
  u32 v[K];
#pragma unroll
  for (int j = 0; j < K; ++j) {
    const u32 I = t + (u32)(j * GW);
    v[j] = I < (u32)NS ? lane_base(e, xq, s_minv, R, wb, I) : 0u;
  }
  Pat<P0, 0, NS>::template spread<GW>(rho, v, t);
}

struct SieveArgs {
  const DevEngine* engines;
  const DevItem* items;
  const u64* task_prefix;  // [nitems + 1] for this kernel's items
  const u32* item_index;   // [nitems] global item index of each entry
  u32 nitems;
  u32 pad;
  u64 ntask;
  const u32* xq;
  u64* cand_key;
  u32* cand_item;
  u64 cand_cap;
  DevCounters* ctr;
  unsigned long long* task_ctr;
  u32 warp_queue;     // compaction: warp queues below this go one
                      // candidate per warp
  u32 seg_per_task;   // marking: segments per task
};

// The entry of the item holding task t: the last i with task_prefix[i] <=
// t, searched forward from `from` (a CTA's claims only grow, so its next
// task's item is at or after its last one): a few steps, then bisection.
__device__ __forceinline__ u32 task_item(const SieveArgs& a, u64 t, u32 from) {
  u32 lo = from;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (lo + 1 < a.nitems && a.task_prefix[lo + 1] <= t) ++lo;
    else return lo;
  }
  u32 hi = a.nitems;
  while (hi - lo > 1) {
    const u32 mid = (lo + hi) >> 1;
    if (a.task_prefix[mid] <= t) lo = mid; else hi = mid;
  }
  return lo;
}

// Per-warp candidate queues of line offsets v = u * M + R.  A queue
// outlives its warp's blocks and tasks: it is drained when it is full and
// when the CTA moves to another item.  In front of it every thread has a
// column of kColSlots codes (word of the chain << 6 | bit): pushing a
// pattern survivor there takes a store and no vote, and a warp's columns
// are turned into offsets a row at a time, when one is full or the block
// ends.
constexpr u32 kWarps = kBlock / 32;
constexpr u32 kWq = 384;
constexpr u32 kColSlots = 16;

struct SieveSmem {
  u64 queue[kWarps * kWq];
  unsigned short col[kWarps * kColSlots * 32];
  // the first kStaged test primes: every drain starts on these, and a
  // shared load answers in a tenth of the time of one from L2
  TestRec srec[kStaged];
  u32 skq[kStaged];
  u32 sboff[kStaged];     // Dickson: the prime's first word in sbit
  u32 sbit[kStagedBits];  // bit h: min(r, q - r) = h is killed
  TestCtx ctx;            // the current item's tests
  const u32* rounds;
  u32 NP, kind, deep;
  u32 wnext[2];           // next warp block of the current / next CTA task
  u64 task[2];
  u32 item[2];
  u32 minv[kNSMax];
  u32 sbits[kSbits + 1];
  u32 eng;
  u32 status;
  unsigned long long mbar;
};

// Shared bytes of the first NS pattern primes' tables (the prefix a kernel
// variant stages), padded to 16 bytes.
template <int P0, int NS = kNS>
__host__ __device__ constexpr u32 pat_bytes() {
  return ((fk_pat_prefix(P0, NS) + 1) / 2) * 16;
}

// A warp's n candidates against the primes [at, end), 32 at a time: each
// lane holds one prime, every candidate is tested against all of them at
// once and the survivors are compacted in place; the next 32 primes' loads
// are in flight meanwhile.  Returns the survivors' count.
template <int KIND>
__device__ __forceinline__ u32 drain_groups(u64* Q, u32 n, const TestCtx& c,
                                            u32 at, u32 end, u32& ntest) {
  const u32 lane = threadIdx.x & 31;
  if (n == 0 || at >= end) return n;
  Prime<KIND> p, next;
  p.load(c, min(at + lane, end - 1));  // past the end: the last prime again
  for (;;) {
    at += 32;
    next.load(c, min(at + lane, end - 1));
    u32 out = 0;
    for (u32 idx = 0; idx < n; idx += 2) {
      const bool two = idx + 1 < n;
      const u64 v = Q[idx], w = Q[two ? idx + 1 : idx];
      const u32 vl = (u32)v & ((1u << kRedcSplit) - 1u);
      const u32 vh = (u32)(v >> kRedcSplit);
      const u32 wl = (u32)w & ((1u << kRedcSplit) - 1u);
      const u32 wh = (u32)(w >> kRedcSplit);
      const bool kv = p.kills(c, vl, vh), kw = p.kills(c, wl, wh);
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
    ntest += n;
    __syncwarp();
    n = out;
    if (at >= end || n == 0) return n;
    p = next;
  }
}

// Drain one warp's queue of n candidates in place.  Over the first primes
// past the pattern (the staged ones, which kill most): rounds with one
// candidate per lane, the survivors compacted by ballot after each.  Once
// fewer than a.warp_queue are left, or the staged primes are done, the
// candidates share the warp instead: each lane holds one prime and every
// candidate is tested against the warp's 32 primes at once, so no lane
// idles behind a dead candidate and the records of 32 primes are loaded
// (one group ahead) once for all of them.  The survivors go to the global
// list.  Warp-synchronous: every lane calls it with the same n.  Returns
// the lane's prime tests.  Not inlined: the pattern loop around it keeps
// its NS table indexes in registers and runs between drains.
template <int KIND>
__device__ __noinline__ u32 warp_drain(u64* Q, u32 n, const SieveSmem& S,
                                       u32 gitem, u32 wq_short, u64* cand_key,
                                       u32* cand_item, u64 cand_cap,
                                       DevCounters* ctr) {
  const u32 lane = threadIdx.x & 31;
  const u32 lt = (1u << lane) - 1u;
  const TestCtx c = S.ctx;
  const u32 NP = S.NP, first = __ldg(S.rounds);
  const u32 nstaged = min(kStaged, NP - first);
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
        bool kill = false;
#pragma unroll
        for (u32 j = 0; j < kRoundUnroll; ++j) {
          const TestRec t = S.srec[i + j];
          const u32 q = redc_residue(t, S.skq[i + j], vl, vh);
          if (KIND == KIND_DICKSON) {
            const u32 h = min(q, t.q - q);
            kill |= (S.sbit[S.sboff[i + j] + (h >> 5)] >> (h & 31)) & 1u;
          } else {
            kill |= kill_test<KIND>(c, first + i + j, t, q);
          }
        }
        alive = alive && !kill;
      }
      const u32 bal = __ballot_sync(0xffffffffu, alive);
      if (alive) Q[out + __popc(bal & lt)] = v;  // out <= base: read already
      out += __popc(bal);
    }
    __syncwarp();
    n = out;
  }
  at = min(first + at, NP);
  const u32 deep = min(max(S.deep, at), NP);
  n = drain_groups<KIND>(Q, n, c, at, deep, ntest);
  // kDeep groups at a time: fewer votes and more loads in flight, once few
  // candidates die among 128 primes
  constexpr u32 kDeep = KIND == KIND_DICKSON ? 2 : 4;
  at = deep;
  for (; n > 0 && at + 32 * kDeep <= NP; at += 32 * kDeep) {
    Prime<KIND> p[kDeep];
#pragma unroll
    for (u32 j = 0; j < kDeep; ++j) p[j].load(c, at + 32 * j + lane);
    u32 out = 0;
    for (u32 idx = 0; idx < n; ++idx) {
      const u64 v = Q[idx];
      const u32 vl = (u32)v & ((1u << kRedcSplit) - 1u);
      const u32 vh = (u32)(v >> kRedcSplit);
      bool kill = false;
#pragma unroll
      for (u32 j = 0; j < kDeep; ++j) kill |= p[j].kills(c, vl, vh);
      if (!__any_sync(0xffffffffu, kill)) {
        if (lane == 0) Q[out] = v;  // out <= idx: read already
        ++out;
      }
    }
    ntest += kDeep * n;
    __syncwarp();
    n = out;
  }
  n = drain_groups<KIND>(Q, n, c, at, NP, ntest);
  // survivors: one atomic per warp
  if (n) {
    u64 base = 0;
    if (lane == 0) base = atomicAdd(&ctr->ncand, (unsigned long long)n);
    base = __shfl_sync(0xffffffffu, base, 0);
    for (u32 idx = lane; idx < n; idx += 32) {
      if (base + idx < cand_cap) {
        cand_key[base + idx] = Q[idx];
        cand_item[base + idx] = gitem;
      } else {
        atomicOr(&ctr->overflow, 1u);
      }
    }
  }
  __syncwarp();
  return ntest;
}

__device__ __forceinline__ u32 drain_any(u64* Q, u32 n, const SieveSmem& S,
                                         u32 gitem, const SieveArgs& a) {
  if (n == 0) return 0;
  switch (S.kind) {
    case KIND_EULER:
      return warp_drain<KIND_EULER>(Q, n, S, gitem, a.warp_queue, a.cand_key,
                                    a.cand_item, a.cand_cap, a.ctr);
    case KIND_DICKSON:
      return warp_drain<KIND_DICKSON>(Q, n, S, gitem, a.warp_queue, a.cand_key,
                                      a.cand_item, a.cand_cap, a.ctr);
    default:
      return warp_drain<KIND_AP>(Q, n, S, gitem, a.warp_queue, a.cand_key,
                                 a.cand_item, a.cand_cap, a.ctr);
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
template <int P0, int NS>
__device__ __forceinline__ bool stage_patterns(u64* spat, const DevEngine& eg,
                                               unsigned long long* mbar,
                                               u32* status, u32& phase,
                                               DevCounters* ctr) {
  __syncthreads();
  if (threadIdx.x == 0) {
    *status = 0;
    const u32 mb = smem_u32(mbar);
    const u32 bytes = pat_bytes<P0, NS>();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile(
        "mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb),
        "r"(bytes)
        : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1], %2, [%3];" ::"r"(smem_u32(spat)),
        "l"((u64)__cvta_generic_to_global(eg.pat)), "r"(bytes), "r"(mb)
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
// holds qn entries and is drained when a row may not fit.  The thread's
// chain: lane R, words w0, w0 + G, ...  Returns the queue's new length and
// adds the lane's prime tests to ntest.  Not inlined, as warp_drain.
static __device__ __noinline__ u32 flush_columns(const SieveSmem& S, u64* Q,
                                          const unsigned short* C, u32 qn,
                                          u32 cn, u64 R, u64 M, u32 w0, u32 G,
                                          u32 gitem, const SieveArgs& a,
                                          u32* ntest) {
  const u32 wl = threadIdx.x & 31;
  const u32 rows = __reduce_max_sync(0xffffffffu, cn);
  for (u32 r = 0; r < rows; ++r) {
    const u32 bal = __ballot_sync(0xffffffffu, r < cn);
    if (qn + 32 > kWq) {
      *ntest += drain_any(Q, qn, S, gitem, a);
      qn = 0;
    }
    if (r < cn) {
      const u32 code = C[32 * r];
      const u64 u = 64ull * (w0 + (code >> 6) * G) + (code & 63u);
      Q[qn + __popc(bal & ((1u << wl) - 1u))] = u * M + R;
    }
    qn += __popc(bal);
  }
  __syncwarp();
  return qn;
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

// One block of 32 threads' chains: thread wl of the warp sweeps chain
// gw + (wl >> gsh) of the item and pushes its pattern survivors through its
// column into the warp's queue (qn entries).
template <int P0, int NS>
__device__ __forceinline__ void sieve_block(
    const u64* __restrict__ spat, SieveSmem& S, u64* Q, u32& qn,
    const SieveArgs& a, const DevEngine& e, const DevItem& it, u32 gitem,
    u64 gw, u64 nchain, u32& ntest, u32& nword) {
  const u32 wl = threadIdx.x & 31;
  const u32 G = it.lane_threads;
  const u32 gsh = G == 32 ? 5u : (G == 8 ? 3u : 0u);
  const u32 Tc = it.Tc, L = e.L;
  const u64 U = it.U, M = e.M;
  // ---- this thread's chain -----------------------------------------
  const u64 g = gw + (wl >> gsh);
  const bool active = g < nchain;
  u32 chunk = 0, lane = 0;   // chunks per lane: below 2^30 words
  if (active) {
    if (nchain <= 0xFFFFFFFFull) {
      chunk = (u32)g / L;
      lane = (u32)g - chunk * L;
    } else {
      chunk = (u32)(g / L);
      lane = (u32)(g % L);
    }
  }
  const u64 R = active ? e.lanes[lane] : 0;
  const u32 w0 = chunk * (G * Tc) + (wl & (G - 1));
  const u32* xq = a.xq + it.xq_off;
  u32 rho[NS];
  if (G == 32) {
    // the whole warp sweeps one lane: thread I works out prime I's base
    // index once and the warp shares it (instead of every thread
    // computing all NS of them)
    shared_setup<P0, NS, 32>(rho, e, xq, S.minv, R, chunk * 32ull * Tc, wl);
  } else if (G == 8) {
    // the same within each group of eight threads sweeping one lane
    shared_setup<P0, NS, 8>(rho, e, xq, S.minv, R, chunk * 8ull * Tc, wl & 7u);
  } else {
    Pat<P0, 0, NS>::setup(rho, R, 64ull * w0, xq, S.minv);
  }
  unsigned short* C = S.col + (threadIdx.x >> 5) * (kColSlots * 32) + wl;
  u32 cn = 0;
  // words in range: below wend; words from 1 to wfull - 1 lie whole inside
  // the item, so only the first word (lo_off) and the last (hi_last, U)
  // need a validity mask
  const u32 wend = (u32)((U + 63) >> 6);
  const u32 wfull = U ? (u32)((U - 1) >> 6) : 0;
  if (active && w0 < wend) nword += min(Tc, (wend - w0 + G - 1) / G);
  for (u32 wi = 0; wi < Tc; wi += 2) {
    // two words of the chain: j = wi and wi + 1
    u64 acc[4] = {0, 0, 0, 0};
    if (G == 32)
      Pat<P0, 0, NS>::template word2<32>(spat, rho, acc);
    else if (G == 8)
      Pat<P0, 0, NS>::template word2<8>(spat, rho, acc);
    else
      Pat<P0, 0, NS>::template word2<1>(spat, rho, acc);
    u64 sv[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const u32 w = w0 + (wi + k) * G;
      u64 s = ~(acc[k * 2] | acc[k * 2 + 1]);
      if (!active || wi + k >= Tc || w >= wend) {
        s = 0;
      } else if (w == 0 || w >= wfull) {
        const u64 left = U - 64ull * w;
        if (left < 64) s &= (1ull << left) - 1ull;
        if (w == 0 && R < it.lo_off) s &= ~1ull;
        if (left <= 64 && R >= it.hi_last) s &= ~(1ull << (left - 1));
      }
      sv[k] = s;
    }
    // into the columns; a full one empties the warp's
    u32 x[4] = {(u32)sv[0], (u32)(sv[0] >> 32), (u32)sv[1],
                (u32)(sv[1] >> 32)};
    for (;;) {
#pragma unroll
      for (int k = 0; k < 4; ++k) push_half(x[k], (wi << 6) + 32 * k, C, cn);
      if (!__any_sync(0xffffffffu, (x[0] | x[1] | x[2] | x[3]) != 0)) break;
      // the table indexes wait out the flush in local memory: live across
      // the call they would be spilled in the word loop instead
      volatile u32 keep[NS];
#pragma unroll
      for (int i = 0; i < NS; ++i) keep[i] = rho[i];
      qn = flush_columns(S, Q, C, qn, cn, R, M, w0, G, gitem, a, &ntest);
      cn = 0;
#pragma unroll
      for (int i = 0; i < NS; ++i) rho[i] = keep[i];
    }
  }
  // the codes refer to this block's chains
  qn = flush_columns(S, Q, C, qn, cn, R, M, w0, G, gitem, a, &ntest);
}

// Claim the CTA's next task into slot p: its number and its item (entry of
// the family's list).
__device__ __forceinline__ void claim_task(const SieveArgs& a, SieveSmem& S,
                                           u32 p, u32 from) {
  const u64 t = atomicAdd(a.task_ctr, 1ull);
  S.task[p] = t;
  S.wnext[p] = 0;
  S.item[p] = t < a.ntask ? task_item(a, t, from) : 0u;
}

// NS: the pattern primes this variant stages (the engine descriptor's NS
// and round cuts must match it).  A CTA task is it.blocks blocks of 32
// threads' chains, claimed by the warps from the CTA's counter, so a warp
// held up by a queue drain takes fewer of them; the next task is claimed
// while this one runs, so a task costs one barrier.
template <int P0, int NS>
__global__ void __launch_bounds__(kBlock, 3)
    k_sieve(const __grid_constant__ SieveArgs a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  u64* spat = reinterpret_cast<u64*>(smem_raw);
  SieveSmem& S = *reinterpret_cast<SieveSmem*>(smem_raw + pat_bytes<P0, NS>());
  const u32 tid = threadIdx.x, wl = tid & 31, wid = tid >> 5;
  if (tid == 0) {
    S.eng = 0xFFFFFFFFu;
    const u32 mb = smem_u32(&S.mbar);
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb)
                 : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    claim_task(a, S, 0, 0);
  }
  __syncthreads();
  u32 phase = 0;
  u64* Q = S.queue + wid * kWq;
  u32 qn = 0, gitem = 0xFFFFFFFFu;
  u32 ntest = 0, nword = 0;  // since the last report
  for (u32 p = 0;; p ^= 1u) {
    const u64 task = S.task[p];
    const u32 entry = S.item[p];
    const bool done = task >= a.ntask;
    const u32 next = done ? 0xFFFFFFFFu : a.item_index[entry];
    if (done || next != gitem) {
      // another item, or the end (a CTA may find every task claimed before
      // its first): drain this one's queue and report
      ntest += drain_any(Q, qn, S, gitem, a);
      qn = 0;
      u64 nt = ntest, nw = nword;  // warp sums in 64 bits
      ntest = nword = 0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        nt += __shfl_down_sync(0xffffffffu, nt, o);
        nw += __shfl_down_sync(0xffffffffu, nw, o);
      }
      if (wl == 0) {
        if (nt) atomicAdd(&a.ctr->s2_tests, (unsigned long long)nt);
        if (nw) atomicAdd(&a.ctr->s1_words, (unsigned long long)nw);
      }
      if (done) break;
      __syncthreads();   // every warp is past the old item's tables
      gitem = next;
      const u32 eidx = a.items[gitem].engine;
      const DevEngine& eg = a.engines[eidx];
      if (S.eng != eidx) {
        // ---- engine switch: stage its pattern table into shared memory ----
        if (!stage_patterns<P0, NS>(spat, eg, &S.mbar, &S.status, phase, a.ctr))
          return;
        for (u32 i = tid; i < (u32)NS; i += kBlock) S.minv[i] = eg.pat_minv[i];
        for (u32 i = tid; i <= eg.sbits_words; i += kBlock)
          S.sbits[i] = i < eg.sbits_words ? eg.sbits[i] : 0u;
        __syncthreads();   // and every warp has read S.eng
        if (tid == 0) S.eng = eidx;
      }
      const u32 first = eg.rounds[0];
      if (tid < (u32)kStaged && first < eg.NP) {
        const u32 p = min(first + tid, eg.NP - 1);  // past the end: the last
        S.srec[tid] = eg.trec[p];
        S.skq[tid] = a.xq[a.items[gitem].xq_off + p];
        if (eg.kind == KIND_DICKSON)
          S.sboff[tid] = eg.boff[p - kNSMin] - eg.boff[first - kNSMin];
      }
      if (eg.kind == KIND_DICKSON && first < eg.NP) {
        const u32 b0 = eg.boff[first - kNSMin];
        const u32 b1 = eg.boff[min(first + kStaged, eg.NP) - kNSMin];
        for (u32 i = b0 + tid; i < b1; i += kBlock) S.sbit[i - b0] = eg.bits[i];
      }
      if (tid == 0) {
        S.ctx = TestCtx{eg.trec, eg.filt, a.xq + a.items[gitem].xq_off,
                        eg.lists, S.sbits, eg.n, eg.xxmax, eg.sbits_words,
                        eg.ap_div};
        S.rounds = eg.rounds;
        S.NP = eg.NP;
        S.deep = eg.deep;
        S.kind = eg.kind;
      }
      __syncthreads();
    }
    if (tid == 0) claim_task(a, S, p ^ 1u, entry);
    const DevItem& it = a.items[gitem];
    const DevEngine& e = a.engines[it.engine];
    const u32 G = it.lane_threads, nblock = it.blocks;
    const u32 cpw = G == 32 ? 1u : (G == 8 ? 4u : 32u);  // chains per block
    const u64 nchain = it.nchunk * e.L;
    const u64 b0 = (task - a.task_prefix[entry]) * (u64)nblock;
    for (;;) {
      u32 wt = 0;
      if (wl == 0) wt = atomicAdd(&S.wnext[p], 1u);
      wt = __shfl_sync(0xffffffffu, wt, 0);
      if (wt >= nblock) break;
      const u64 gw = (b0 + wt) * cpw;      // the block's first chain
      if (gw >= nchain) break;             // and every later one's too
      sieve_block<P0, NS>(spat, S, Q, qn, a, e, it, gitem, gw, nchain, ntest,
                          nword);
    }
    __syncthreads();   // the next task is claimed, this one's counter free
  }
}

}  // namespace fk
