// fk_classify.cuh -- base residues, chain classification and ordering.
//
// k_xq        X0 mod q, or its multiple, for every (item, sieve prime): the per-launch
//             "(k_base mod q)" tables of the reference
//             (euler-prime-runs/euler_gpu.py:1474-1477,
//             primorial-ap/ap_gpu.py:586-593), computed on the device from
//             the 128-bit base.
// k_dense     fills the candidate list with every x of a DENSE item (the
//             launchers' low passes below the engine floors).
// k_classify, k_exact
//             the on-device SPRP stage: each candidate's chain depth by
//             the reference's definition for its engine (Euler
//             mr_run_length, Dickson run_length / sprp_run, AP two-pass
//             chain_depth), kept when it reaches the item's threshold.
// k_order_prep, k_bucket_*, k_scan, k_sort_seg
//             order the kept entries per item ascending in x without a
//             host sort: counting scatter by item, then a bitonic sort of
//             each item's segment.
#pragma once
#include "fk_sieve.cuh"
#include "fk_sprp.cuh"
#include "fk_types.h"

namespace fk {

struct ClassArgs {
  const DevEngine* engines;
  const DevItem* items;
  const u64* cand_key;
  const u32* cand_item;
  u64 cand_cap;
  DevCounters* ctr;
  OutRec* out;
  u64 out_cap;
  u32* item_count;
  u64* exact;               // [cand_cap] candidate index << 8 | base-2 depth
  u64 spec_lanes;           // lanes worth filling with a candidate's values
};

__device__ __forceinline__ void emit_out(const ClassArgs& a, u32 item,
                                         u64 packed) {
  const unsigned long long p = atomicAdd(&a.ctr->nout, 1ull);
  if (p < a.out_cap) {
    a.out[p].packed = packed;
    a.out[p].item = item;
    atomicAdd(a.item_count + item, 1u);
  } else {
    atomicOr(&a.ctr->overflow, 2u);
  }
}

// The values of one candidate's chain (Euler x^2 + x + p for x = t, Dickson
// (t + 1) * k^2 + 1, AP p + t * d).
struct Chain {
  u32 kind;
  u128 x;   // Euler / AP: p
  V3 kk;    // Dickson: k^2
  V3 d;     // AP: difference
};

__device__ __forceinline__ V3 chain_value(const Chain& c, u32 t) {
  if (c.kind == KIND_EULER) return v3_from_u128(c.x + (u128)((u64)t * t + t));
  if (c.kind == KIND_DICKSON) {
    V3 v = v3_mul_u64(c.kk, (u64)(t + 1));
    const V3 one = {{1, 0, 0}};
    return v3_add(v, one);
  }
  return v3_add(v3_from_u128(c.x), v3_mul_u64(c.d, (u64)t));
}

// First t < lim whose value fails sprp_base2 (lim when none does): an
// upper bound on every engine's depth, because mr_is_prime implies
// sprp_base2 (huntlib/primes.py:38-46 tests base 2 first).
__device__ u32 chain_base2(const Chain& c, u32 lim, u64* imad, u64* nval) {
  u32 t = 0;
  while (t < lim) {
    ++*nval;
    if (!sprp(chain_value(c, t), true, imad)) break;
    ++t;
  }
  return t;
}

// Every value below d2 passed base 2; the exact mr_is_prime chain ends at
// the first of them that fails one of the other six bases.
__device__ u32 chain_exact(const Chain& c, u32 d2, u64* imad, u64* nval) {
  u32 t = 0;
  while (t < d2) {
    ++*nval;
    if (!sprp_rest(chain_value(c, t), imad)) break;
    ++t;
  }
  return t;
}

// Depth by the reference's definition for the engine, or -1 when the
// base-2 bound already proves it below the threshold:
//   Euler    mr_run_length (euler_search.py:258-262), searched to
//            max(threshold, cap); hunt keeps f >= threshold, reports
//            min(f, cap); the dense low pass keeps min(f, cap) >= thr
//   Dickson  run_length (ladder_search.py:143-148), or the launcher's
//            two-pass sprp_run (dickson-ladders/launch.py:310-343)
//   AP       two-pass chain_depth (ap_search.py:160-194)
__device__ int chain_depth_thr(const Chain& c, u32 mode, u32 thr, u32 cap,
                               bool two_pass, u64* imad, u64* nval) {
  if (c.kind == KIND_EULER) {
    const u32 lim = max(thr, cap);
    const u32 d2 = chain_base2(c, lim, imad, nval);
    const bool dense = mode == MODE_DENSE;
    if ((dense ? min(d2, cap) : d2) < thr) return -1;
    const u32 f = chain_exact(c, d2, imad, nval);
    const u32 depth = min(f, cap);
    return ((dense ? depth : f) >= thr) ? (int)depth : -1;
  }
  const u32 d2 = chain_base2(c, cap, imad, nval);
  const u32 pass = (c.kind == KIND_AP) ? 6u : (two_pass ? 5u : 0u);
  u32 depth;
  if (d2 < pass) {
    depth = d2;
  } else {
    if (d2 < thr) return -1;
    depth = chain_exact(c, d2, imad, nval);
  }
  return depth >= thr ? (int)depth : -1;
}

// The SPRP stage, in two kernels.
//
// k_classify finds each candidate's base-2 depth d2 -- the first t whose
// value fails the strong test to base 2, an upper bound on every engine's
// depth (mr_is_prime implies sprp_base2) -- and decides by the engine's
// rules (chain_depth_thr): dropped when d2 already proves it below the
// threshold, reported for the two-pass engines below their exact-from depth,
// else put on the exact list with its d2.  k_exact then tests the values t <
// d2 of the listed candidates to the six other bases: all 6 * d2 tests of a
// candidate are independent, so a warp's lanes share them out instead of one
// lane running them one after the other (which alone took 0.6 ms of an 0.78
// ms hunt of 32 candidates, at 6 of 32 lanes active).
//
// In k_classify a chain of G lanes tests G consecutive values of one
// candidate at once when the candidates are too few to fill the chip (G up
// to 32: the tests past the first failure cost nothing there).  With G = 1
// it is a step interpreter: each lane holds the state of one candidate and
// performs exactly one strong test per step, and a lane whose candidate is
// finished takes the next one at once from a chunk its warp fetched, so a
// warp never waits for its longest chain.
struct LaneState {
  Chain c;
  u64 v, i;
  u32 item, mode, thr, cap;
  u32 t, lim, pass;
};

// The chain of candidate i's value at line offset v of item `item`; false
// when a Dickson square does not fit 192 bits.
__device__ __forceinline__ bool chain_init(Chain& c, const ClassArgs& a,
                                           const DevItem& it,
                                           const DevEngine& e, u64 v) {
  c.kind = e.kind;
  c.x = (((u128)it.X0_hi << 64) | it.X0_lo) + v;
  if (e.kind == KIND_DICKSON) {
    const u64 W = (it.mode == MODE_DENSE) ? 1ull : e.W;
    bool of = false;
    const u128 k = c.x * (u128)W;
    c.kk = v3_mul_128(k, k, &of);
    if (of) {
      atomicOr(&a.ctr->overflow, 8u);
      return false;
    }
  } else if (e.kind == KIND_AP) {
    c.d = V3{{e.d_lo, e.d_hi, 0}};
  }
  return true;
}

__device__ __forceinline__ bool lane_init(LaneState& s, const ClassArgs& a,
                                          u64 i, bool emit) {
  s.i = i;
  s.item = a.cand_item[i];
  const DevItem& it = a.items[s.item];
  const DevEngine& e = a.engines[it.engine];
  s.v = a.cand_key[i];
  s.mode = it.mode;
  if (s.mode == MODE_SIEVE) {
    if (emit) emit_out(a, s.item, s.v << 8);
    return false;
  }
  s.thr = it.threshold;
  s.cap = it.cap;
  if (!chain_init(s.c, a, it, e, s.v)) return false;
  s.pass = (e.kind == KIND_AP) ? 6u
           : (e.kind == KIND_DICKSON ? (e.two_pass ? 5u : 0u) : 0u);
  s.lim = (e.kind == KIND_EULER) ? max(s.thr, s.cap) : s.cap;
  s.t = 0;
  return true;
}

// Finish with the exact depth: emit when it reaches the threshold.
__device__ __forceinline__ void emit_final(const ClassArgs& a, u32 kind,
                                           u32 mode, u32 thr, u32 cap,
                                           u32 item, u64 v, u32 exact) {
  if (kind == KIND_EULER) {
    const u32 depth = min(exact, cap);
    const u32 test = (mode == MODE_DENSE) ? depth : exact;
    if (test >= thr) emit_out(a, item, (v << 8) | (u64)min(depth, 255u));
  } else if (exact >= thr) {
    emit_out(a, item, (v << 8) | (u64)min(exact, 255u));
  }
}

// After the base-2 chain of depth d2: report it, drop it, or list it for
// the exact tests.
__device__ __forceinline__ void lane_decide(const LaneState& s,
                                            const ClassArgs& a, u32 d2) {
  if (s.c.kind == KIND_EULER) {
    const u32 bound = (s.mode == MODE_DENSE) ? min(d2, s.cap) : d2;
    if (bound < s.thr) return;
  } else {
    if (d2 < s.pass) {
      if (d2 >= s.thr) emit_out(a, s.item, (s.v << 8) | (u64)min(d2, 255u));
      return;
    }
    if (d2 < s.thr) return;
  }
  if (d2 == 0) {
    emit_final(a, s.c.kind, s.mode, s.thr, s.cap, s.item, s.v, 0);
    return;
  }
  // at most one entry per candidate, so the list never overflows
  a.exact[atomicAdd(&a.ctr->nexact, 1ull)] = (s.i << 8) | (u64)d2;
}

// One atomic per warp for the work counters.
__device__ __forceinline__ void report_work(const ClassArgs& a, u64 imad,
                                            u64 nval) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    imad += __shfl_down_sync(0xffffffffu, imad, o);
    nval += __shfl_down_sync(0xffffffffu, nval, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (imad) atomicAdd(&a.ctr->imad_alg, (unsigned long long)imad);
    if (nval) atomicAdd(&a.ctr->sprp_values, (unsigned long long)nval);
  }
}

__global__ void __launch_bounds__(kBlock) k_classify(ClassArgs a) {
  u64 n = a.ctr->ncand;
  if (n > a.cand_cap) n = a.cand_cap;
  const u32 lane = threadIdx.x & 31;
  const u32 lt = (1u << lane) - 1u;
  LaneState st;
  u64 imad = 0, nval = 0;
  // lanes per candidate: the most that keep every lane's warp resident with
  // few enough others that a step takes no longer than it takes alone
  u32 G = 32;
  while (G > 1 && n * G > a.spec_lanes) G >>= 1;
  if (G > 1) {
    const u32 gl = lane & (G - 1), g0 = lane & ~(G - 1);
    const u32 gmask = (G == 32 ? 0xffffffffu : ((1u << G) - 1u)) << g0;
    const u64 groups = (u64)gridDim.x * (kBlock / G);
    // consecutive candidates go to different CTAs.  The whole warp stays in
    // the loop while one of its groups has a candidate, so the votes are
    // warp-wide
    for (u64 i = ((u64)(threadIdx.x >> 5) * gridDim.x + blockIdx.x) * (32 / G) +
                 lane / G;
         __any_sync(0xffffffffu, i < n); i += groups) {
      bool active = i < n && lane_init(st, a, i, gl == 0);
      while (__any_sync(0xffffffffu, active)) {
        const u32 t = st.t + gl;
        bool fail = false;
        if (active && t < st.lim) {
          ++nval;
          fail = !sprp_step(chain_value(st.c, t), 0, &imad);
        }
        const u32 bad = __ballot_sync(0xffffffffu, fail) & gmask;
        if (active) {
          if (bad || st.t + G >= st.lim) {
            if (gl == 0)
              lane_decide(st, a,
                          bad ? st.t + __ffs((int)bad) - 1 - g0 : st.lim);
            active = false;
          } else {
            st.t += G;
          }
        }
      }
    }
    report_work(a, imad, nval);
    return;
  }
  u64 chunk_pos = 0, chunk_end = 0;  // warp-uniform
  bool active = false, drained = false;
  for (;;) {
    // hand new candidates to idle lanes
    while (!drained) {
      const u32 idle = __ballot_sync(0xffffffffu, !active);
      if (!idle) break;
      if (chunk_pos >= chunk_end) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(&a.ctr->class_next, (u64)kClassChunk);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= n) {
          drained = true;
          break;
        }
        chunk_pos = base;
        chunk_end = min(base + (u64)kClassChunk, n);
      }
      const u32 rank = __popc(idle & lt);
      const u32 take = (u32)min((u64)__popc(idle), chunk_end - chunk_pos);
      if (!active && rank < take)
        active = lane_init(st, a, chunk_pos + rank, true);
      chunk_pos += take;
    }
    if (__ballot_sync(0xffffffffu, active) == 0) break;
    if (active) {
      bool pass = false;
      if (st.lim > 0) {
        ++nval;
        pass = sprp_step(chain_value(st.c, st.t), 0, &imad);
      }
      if (pass && st.t + 1 < st.lim) {
        ++st.t;
      } else {
        lane_decide(st, a, pass ? st.lim : st.t);
        active = false;
      }
    }
  }
  report_work(a, imad, nval);
}

// The exact tests: a warp takes up to kExactChunk listed candidates and its
// lanes share out all their (value, base) tests in order; a failure lowers
// the candidate's depth to the value's index.
constexpr u32 kExactChunk = 16;
__global__ void __launch_bounds__(kBlock) k_exact(ClassArgs a) {
  __shared__ u32 s_first[kBlock / 32][kExactChunk];
  const u64 n = a.ctr->nexact;
  const u32 lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  u32* first = s_first[wid];
  u64 imad = 0, nval = 0;
  // fewer at a time when they are too few to go round
  const u64 warps = (u64)gridDim.x * (kBlock / 32);
  const u32 chunk =
      (u32)min((u64)kExactChunk, max((u64)1, n / (warps * 2)));
  for (;;) {
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(&a.ctr->exact_next, (u64)chunk);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= n) break;
    const u32 m = (u32)min((u64)chunk, n - base);
    const u64 rec = lane < m ? a.exact[base + lane] : 0;
    const u32 d2 = (u32)(rec & 255u);
    if (lane < m) first[lane] = d2;
    u32 end = 6 * d2;   // inclusive prefix of the test counts
#pragma unroll
    for (int o = 1; o < (int)kExactChunk; o <<= 1) {
      const u32 y = __shfl_up_sync(0xffffffffu, end, o);
      if (lane >= (u32)o) end += y;
    }
    const u32 total = __shfl_sync(0xffffffffu, end, m - 1);
    __syncwarp();
    for (u32 k0 = 0; k0 < total; k0 += 32) {
      const u32 k = k0 + lane;
      // the candidate of test k: the first whose prefix passes k
      u32 c = 0, from = 0;
      for (u32 j = 0; j < m; ++j) {
        const u32 e = __shfl_sync(0xffffffffu, end, j);
        if (e <= k) {
          c = j + 1;
          from = e;
        }
      }
      const u64 r = __shfl_sync(0xffffffffu, rec, c < m ? c : 0);
      if (k < total) {
        const u32 t = (k - from) / 6u, b = (k - from) % 6u + 1u;
        const u64 i = r >> 8;
        const DevItem& it = a.items[a.cand_item[i]];
        Chain ch;
        chain_init(ch, a, it, a.engines[it.engine], a.cand_key[i]);
        ++nval;
        if (!sprp_step(chain_value(ch, t), (int)b, &imad))
          atomicMin(&first[c], t);
      }
      __syncwarp();
    }
    if (lane < m) {
      const u64 i = rec >> 8;
      const u32 item = a.cand_item[i];
      const DevItem& it = a.items[item];
      emit_final(a, a.engines[it.engine].kind, it.mode, it.threshold, it.cap,
                 item, a.cand_key[i], first[lane]);
    }
    __syncwarp();
  }
  report_work(a, imad, nval);
}

// Every x of dense items, into the candidate list.
__global__ void k_dense(const DevItem* items, const u32* dense_idx,
                        u32 ndense, u64* cand_key, u32* cand_item,
                        u64 cand_cap, DevCounters* ctr) {
  for (u32 d = 0; d < ndense; ++d) {
    const u32 item = dense_idx[d];
    const u64 cnt = items[item].U;
    for (u64 v = (u64)blockIdx.x * blockDim.x + threadIdx.x; v < cnt;
         v += (u64)gridDim.x * blockDim.x) {
      const unsigned long long p = atomicAdd(&ctr->ncand, 1ull);
      if (p < cand_cap) {
        cand_key[p] = v;
        cand_item[p] = item;
      } else {
        atomicOr(&ctr->overflow, 1u);
      }
    }
  }
}

// The base residues of every (item, prime) of sieve items.
__global__ void k_xq(const DevEngine* engines, const DevItem* items,
                     const u32* sieve_idx, u32 nsieve, u32* xq) {
  for (u32 s = blockIdx.y; s < nsieve; s += gridDim.y) {
    const DevItem it = items[sieve_idx[s]];
    const DevEngine& e = engines[it.engine];
    const u32 n = base_entries(e, it);
    for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x)
      xq[it.xq_off + i] = base_residue(e, it, i);
  }
}

// Exclusive scan of n counts by one CTA of kBlock threads: off[0, n].
template <typename F>
__device__ __forceinline__ u64 cta_scan(u32 n, u64* off, F count) {
  __shared__ u64 s_warp[kBlock / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  u64 carry = 0;
  for (u32 base = 0; base < n; base += kBlock) {
    const u32 i = base + threadIdx.x;
    const u64 v = i < n ? count(i) : 0;
    u64 x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u64 y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[wid] = x;
    __syncthreads();
    u64 pre = 0, tot = 0;
    for (int w = 0; w < kBlock / 32; ++w) {
      pre += (w < wid) ? s_warp[w] : 0;
      tot += s_warp[w];
    }
    if (i < n) off[i] = carry + pre + x - v;
    carry += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) off[n] = carry;
  return carry;
}

// The scan of the bucket counts, their number read from device memory.
__global__ void __launch_bounds__(kBlock) k_scan(const u32* count, u64* off,
                                                 const u32* n_dev) {
  cta_scan(*n_dev, off, [&](u32 i) { return (u64)count[i]; });
}

// Buckets for ordering: every item's entries are split by key range into
// nb = ceil(count / kBucketFill) buckets (the entries of one interval are
// spread over its span, so a bucket holds about kBucketFill of them), and
// each bucket is then sorted on its own (k_sort_seg).  One CTA: each item's
// first output and first bucket, the number of buckets, and their counters
// cleared.
constexpr int kOrderBlock = kBlock;
__global__ void __launch_bounds__(kOrderBlock)
    k_order_prep(const u32* count, u32 nitems, u64* off, u32* nb, u64* bbase,
                 u32* nbuckets, u32* bcount, u32* bfill) {
  cta_scan(nitems, off, [&](u32 i) { return (u64)count[i]; });
  const u64 total = cta_scan(nitems, bbase, [&](u32 i) {
    const u32 k = (count[i] + kBucketFill - 1) / kBucketFill;
    nb[i] = k;
    return (u64)k;
  });
  for (u32 i = threadIdx.x; i < total; i += kBlock) bcount[i] = bfill[i] = 0;
  if (threadIdx.x == 0) *nbuckets = (u32)total;
}

__device__ __forceinline__ u32 bucket_of(const OutRec& r, const DevItem* items,
                                         const DevEngine* engines,
                                         const u64* bucket_base,
                                         const u32* nb) {
  const DevItem it = items[r.item];
  const u64 span = (it.mode == MODE_DENSE)
                       ? it.U
                       : it.U * engines[it.engine].M;  // keys are below U*M
  const u32 k = nb[r.item];
  const u64 key = r.packed >> 8;
  u64 b = (u64)(((u128)key * k) / (span ? span : 1));
  if (b >= k) b = k - 1;
  return (u32)(bucket_base[r.item] + b);
}

__global__ void k_bucket_count(const OutRec* out, const DevCounters* ctr,
                               u64 out_cap, const DevItem* items,
                               const DevEngine* engines,
                               const u64* bucket_base, const u32* nb,
                               u32* bcount) {
  u64 n = ctr->nout;
  if (n > out_cap) n = out_cap;
  for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (u64)gridDim.x * blockDim.x)
    atomicAdd(bcount + bucket_of(out[i], items, engines, bucket_base, nb), 1u);
}

__global__ void k_bucket_scatter(const OutRec* out, const DevCounters* ctr,
                                 u64 out_cap, const DevItem* items,
                                 const DevEngine* engines,
                                 const u64* bucket_base, const u32* nb,
                                 const u64* boff, u32* bfill, u64* sorted) {
  u64 n = ctr->nout;
  if (n > out_cap) n = out_cap;
  for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (u64)gridDim.x * blockDim.x) {
    const OutRec r = out[i];
    const u32 b = bucket_of(r, items, engines, bucket_base, nb);
    sorted[boff[b] + atomicAdd(bfill + b, 1u)] = r.packed;
  }
}

// Bitonic sort of buf[0, npow) ascending, npow a power of two, by one CTA.
__device__ void cta_bitonic(u64* buf, u32 npow) {
  for (u32 k = 2; k <= npow; k <<= 1) {
    for (u32 j = k >> 1; j > 0; j >>= 1) {
      for (u32 i = threadIdx.x; i < npow; i += blockDim.x) {
        const u32 l = i ^ j;
        if (l > i) {
          const u64 x = buf[i], y = buf[l];
          const bool up = (i & k) == 0;
          if ((x > y) == up) {
            buf[i] = y;
            buf[l] = x;
          }
        }
      }
      __syncthreads();
    }
  }
}

// Sort every item's segment of `sorted` (keys unique per item).
__global__ void __launch_bounds__(kBlock) k_sort_seg(
    u64* sorted, const u64* off, const u32* nitems_p, u64* scratch) {
  __shared__ u64 s_buf[kSortSmem];
  const u32 nitems = *nitems_p;
  for (u32 item = blockIdx.x; item < nitems; item += gridDim.x) {
    const u64 o = off[item];
    const u32 n = (u32)(off[item + 1] - o);
    if (n < 2) continue;
    u32 npow = 1;
    while (npow < n) npow <<= 1;
    u64* buf = (npow <= (u32)kSortSmem) ? s_buf : scratch + 2 * o;
    for (u32 i = threadIdx.x; i < npow; i += blockDim.x)
      buf[i] = i < n ? sorted[o + i] : ~0ull;
    __syncthreads();
    cta_bitonic(buf, npow);
    for (u32 i = threadIdx.x; i < n; i += blockDim.x) sorted[o + i] = buf[i];
    __syncthreads();
  }
}

}  // namespace fk
