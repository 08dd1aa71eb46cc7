// fk_mark.cuh -- the marking sieve for long lanes (stage S1 + marking).
//
// A weak sieve (small n: every prime kills only a few residues) leaves many
// candidates alive deep into the prime list, and testing each of them
// against every remaining prime costs tens of tests per candidate.  Long
// lanes are therefore sieved the Eratosthenes way instead: one CTA owns one
// lane over SEG * seg_per_task consecutive periods, and per segment of SEG
// periods (16384, 32768 or 65536: a template variant chosen per batch) it
//   (a) ORs the NS compile-time pattern primes into SEG / 16384 words per
//       thread (the stage-1a pattern sieve of fk_sieve.cuh),
//   (b) marks every other prime below 2^16 into a SEG-byte shared map: plain
//       byte stores (a mark is idempotent: no read-modify-write, no atomic),
//   (c) extracts the periods that neither marked, tests any primes beyond
//       the marked range one by one, and appends the survivors to the
//       candidate list.
// The unit of (b) is a block of 32 primes of one octave, one per lane: a
// lane reads its prime and its offset once and walks the prime's residues,
// two to a coalesced 4-byte load, each a subtraction, a fold and its stores
// -- fixed sequences of predicated stores, no loop, from q >= SEG / 2 on.
// The primes with 16 hits a segment or more go by (prime, residue) pairs, 32
// of nearly equal step to a warp, so the lanes share their trip counts.  A
// whole segment holds floor(SEG / q) hits of every lane at least, and those
// are stored without a bound's test.  The host cuts the work into pieces and
// deals them to the eight warps by cost.  What bounds it: instructions (about
// 25 per 32 residues besides the stores) and the byte stores' bank conflicts
// (32 random bytes take 3.5 wavefronts).  With one 8-byte work entry per
// (prime, residue), dealt to threads at 38 instructions for the two marks of a
// large prime, the marking of 256 mixed intervals took 86.5 ms and this form
// 69 for the same items; the present choice of sieve leaves it fewer, 26 ms.
// Each slot's first hit offset lives in shared memory and steps by the
// tabulated SEG mod q from one segment to the next.
// This is the reference AP engine's bitmap marking (primorial-ap/ap_gpu.py:
// 204-369: tabulated small primes, shared-memory marks for mid primes,
// global atomics for the rest) re-laid out per lane, so no mark needs an
// atomic and every engine kind can use it.
#pragma once
#include "fk_sieve.cuh"

namespace fk {

template <int SEG>
struct MarkSmem {
  unsigned char bytes[SEG];
  unsigned short off16[kMarkSlots];   // first hit offset of each slot's prime
  u32 ph[kNSMax];                     // table index at the segment start
  u32 sbits[kSbits + 1];
  u64 task;
  u32 item;
  u32 eng;
  u32 status;
  u32 pad;
  unsigned long long mbar;
};

// The WPT pattern words of thread t in a segment (words t, t + kBlock, ...:
// a warp's loads are consecutive entries), from each prime's table index at
// the segment start in shared memory: no per-prime index occupies a register
// while the segment is marked.
template <int P0, int I, int NS, int WPT>
struct PatSeg {
  static __device__ __forceinline__ void words(const u64* __restrict__ spat,
                                               const u32* ph, u32 t,
                                               u64* acc) {
    constexpr u32 q = fk_nth_prime(P0 + I);
    constexpr u32 off = fk_pat_prefix(P0, I);
    constexpr u32 st = kBlock % q;
    u32 r = ph[I] + t % q;
    r = min(r, r - q);
#pragma unroll
    for (int k = 0; k < WPT; ++k) {
      acc[k] |= spat[off + r];
      r += st;
      r = min(r, r - q);
    }
    PatSeg<P0, I + 1, NS, WPT>::words(spat, ph, t, acc);
  }
};
template <int P0, int NS, int WPT>
struct PatSeg<P0, NS, NS, WPT> {
  static __device__ __forceinline__ void words(const u64*, const u32*, u32,
                                               u64*) {}
};

template <int MODE>
__device__ __forceinline__ bool tail_alive(u64 v, const DevEngine& e,
                                           const u32* __restrict__ kq,
                                           const u32* s_sbits, u64& ntest) {
  const TestCtx c{e.trec, e.filt, kq, e.lists,
                  e.n, e.xxmax, e.sbits_words, e.ap_div};
  const u32 vl = (u32)v & ((1u << kRedcSplit) - 1u);
  const u32 vh = (u32)(v >> kRedcSplit);
  for (u32 i = e.NPm; i < e.NP; ++i) {
    ++ntest;
    Prime<MODE> p;
    p.load(c, i);
    if (any_kill<MODE, 1>(&p, c, s_sbits, vl, vh))
      return false;
  }
  return true;
}

// Mark one progression in a whole segment: a its first hit of the item,
// step q, K hits without a test and E more with one.  K and E are the same
// in all lanes.  Returns the hits stored.
template <int SEG>
__device__ __forceinline__ u32 mark_many(unsigned char* __restrict__ B, u32 a,
                                         u32 q, u32 K, u32 E) {
  for (u32 c = K >> 2; c > 0; --c, a += 4 * q) {
    B[a] = 1;
    B[a + q] = 1;
    B[a + 2 * q] = 1;
    B[a + 3 * q] = 1;
  }
  if (K & 2u) {
    B[a] = 1;
    B[a + q] = 1;
    a += 2 * q;
  }
  if (K & 1u) {
    B[a] = 1;
    a += q;
  }
  u32 cnt = K;
  for (u32 c = E; c > 0; --c, a += q)
    if (a < SEG) {
      B[a] = 1;
      ++cnt;
    }
  return cnt;
}

// The same below len, in a segment cut short.
__device__ __forceinline__ u32 mark_short(unsigned char* __restrict__ B, u32 a,
                                          u32 q, u32 K, u32 E, u32 len) {
  const u32 end = E ? len : min(len, a + K * q);
  u32 cnt = 0;
  for (; a < end; a += q, ++cnt) B[a] = 1;
  return cnt;
}

// What the marks read besides the map.
struct MarkCtx {
  const unsigned short* off16;   // shared
  const u32* mq;
  const u32* mres;
  u32 qlim, len;                 // len: the segment's periods
};

// The blocks of an item, two residues to a load; mark(a, q) stores the hits
// of the progression a, a + q, ... and returns their count.
template <typename F>
__device__ __forceinline__ u32 mark_blocks(const MarkCtx& c, u32 nblk, u32 f,
                                           u32 block, u32 r0, F mark) {
  const u32 wl = threadIdx.x & 31;
  u32 slot = block * 32 + wl, cnt = 0;
  const u32* res = c.mres + r0 + wl;
  for (; nblk > 0; --nblk, slot += 32) {
    u32 g2 = __ldg(res);
    const u32 q = __ldg(c.mq + slot) & 0xFFFFu, off = c.off16[slot];
    for (u32 j = 0; j < f; j += 2) {
      u32 h0 = (g2 & 0xFFFFu) - off, h1 = (g2 >> 16) - off;
      res += 32;
      if (j + 2 < f) g2 = __ldg(res);
      h0 = min(h0, h0 + q);    // (g - off) mod q: the first hit
      h1 = min(h1, h1 + q);
      if (q >= c.qlim) continue;
      cnt += mark(h0, q);
      if (j + 1 < f) cnt += mark(h1, q);
    }
  }
  return cnt;
}

// K hits and at most E more, in straight line: two instructions a hit
// without a test, four with one.  (The variants stay few and their residue
// loop rolled: the kernel's code has to stay in the instruction cache.  With
// eight residues unrolled the warps waited for instructions, and the marking
// of 256 mixed intervals took 131 ms instead of 69, items as above.)
template <u32 K, u32 E, bool WHOLE>
__device__ __forceinline__ u32 mark_fixed(unsigned char* __restrict__ B,
                                          const MarkCtx& c, const uint4& w) {
  return mark_blocks(c, (w.x >> 8) & 0xFFu, w.x >> 16, w.y, w.z,
                     [&](u32 a, u32 q) {
                       u32 cnt = 0;
                       // a short segment holds few first hits: the
                       // warp mostly leaves here
                       if (!WHOLE && a >= c.len) return cnt;
#pragma unroll
                       for (u32 k = 0; k < K + E; ++k, a += q) {
                         if ((WHOLE && k < K) || a < c.len) {
                           B[a] = 1;
                           ++cnt;
                         }
                       }
                       return cnt;
                     });
}

template <bool WHOLE>
__device__ __forceinline__ u32 mark_fixed_any(unsigned char* __restrict__ B,
                                              const MarkCtx& c, const uint4& w) {
  const bool two = (w.w >> 24) == 2;
  switch ((w.w >> 16) & 0xFFu) {
    case 0: return mark_fixed<0, 1, WHOLE>(B, c, w);
    case 1:
      return two ? mark_fixed<1, 2, WHOLE>(B, c, w)
                 : mark_fixed<1, 1, WHOLE>(B, c, w);
    case 2: return mark_fixed<2, 2, WHOLE>(B, c, w);
    case 3: return mark_fixed<3, 2, WHOLE>(B, c, w);
    case 4: return mark_fixed<4, 2, WHOLE>(B, c, w);
    case 5: return mark_fixed<5, 2, WHOLE>(B, c, w);
    case 6: return mark_fixed<6, 2, WHOLE>(B, c, w);
    default: return mark_fixed<7, 2, WHOLE>(B, c, w);
  }
}

// A warp's items of one segment of len periods (WHOLE: SEG of them).
template <bool WHOLE, int SEG>
__device__ __forceinline__ u32 mark_segment(unsigned char* __restrict__ B,
                                            const unsigned short* off16,
                                            const DevEngine& e, u32 len) {
  const u32 wl = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint4* work = reinterpret_cast<const uint4*>(e.mwork);
  const u32 end = __ldg(e.mwoff + wid + 1);
  u32 i = __ldg(e.mwoff + wid), cnt = 0;
  if (i >= end) return 0;
  const MarkCtx c{off16, e.mq, e.mres, e.qlim, WHOLE ? (u32)SEG : len};
  const u32* mpair = e.mpair;
  const u32 nblock = e.nslots / 32;
  uint4 next = __ldg(work + i);
  while (i < end) {
    const uint4 w = next;
    if (++i < end) next = __ldg(work + i);   // in flight meanwhile
    const u32 kind = w.x & 0xFFu;
    // past the marked range
    if (w.y >= (kind == MARK_PAIRS ? e.qlim : nblock)) continue;
    if (kind == MARK_FIXED) {
      cnt += mark_fixed_any<WHOLE>(B, c, w);
      continue;
    }
    const u32 hit0 = w.w & 0xFFFFu, K = (w.w >> 16) & 0xFFu, E = w.w >> 24;
    // its hits all lie past a short segment's end
    if (!WHOLE && kind == MARK_PAIRS && hit0 * w.y >= len) continue;
    const auto many = [&](u32 h, u32 q) {
      return WHOLE ? mark_many<SEG>(B, h + hit0 * q, q, K, E)
                   : mark_short(B, h + hit0 * q, q, K, E, len);
    };
    if (kind == MARK_PAIRS) {
      const u32 x = __ldg(mpair + w.z + wl), slot = x >> 16;
      const u32 q = __ldg(c.mq + slot) & 0xFFFFu;
      const u32 h = (x & 0xFFFFu) - off16[slot];
      if (q < c.qlim) cnt += many(min(h, h + q), q);
    } else {
      cnt += mark_blocks(c, (w.x >> 8) & 0xFFu, w.x >> 16, w.y, w.z, many);
    }
  }
  return cnt;
}

// The 64 map bytes of word w as bits: four 16-byte loads, their order
// rotated by the thread so that eight lanes at a stride of 64 bytes touch
// all the banks.
__device__ __forceinline__ u64 map_bits(const unsigned char* B, u32 w) {
  const uint4* b = reinterpret_cast<const uint4*>(B + 64 * w);
  const u32 rot = (threadIdx.x >> 1) & 3u;
  u64 m = 0;
#pragma unroll
  for (u32 j = 0; j < 4; ++j) {
    const uint4 x = b[(j + rot) & 3u];   // bytes are 0 or 1
    const u32 k = 0x10204080u;
    const u32 r = ((x.x * k) >> 28) | ((x.y * k) >> 28 << 4) |
                  ((x.z * k) >> 28 << 8) | ((x.w * k) >> 28 << 12);
    m |= (u64)r << (16 * j);
  }
  return rot ? (m << (16 * rot)) | (m >> (64 - 16 * rot)) : m;
}

// NS pattern primes, SEG periods per segment; the engine descriptor's NS
// and marking tables (mq, mwork) must be the ones of this variant.
template <int P0, int NS, int SEG>
__global__ void __launch_bounds__(kBlock, 3) k_mark(SieveArgs a) {
  constexpr int WPT = SEG / (64 * kBlock);  // pattern words per thread
  static_assert(WPT * 64 * kBlock == SEG, "segment must be 1-4 words per thread");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  u64* spat = reinterpret_cast<u64*>(smem_raw);
  MarkSmem<SEG>& S =
      *reinterpret_cast<MarkSmem<SEG>*>(smem_raw + pat_bytes<P0, NS>());
  const int tid = threadIdx.x;
  if (tid == 0) {
    S.eng = 0xFFFFFFFFu;
    const u32 mb = smem_u32(&S.mbar);
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb)
                 : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  u32 phase = 0;
  u64 nmark = 0, ntest = 0, nword = 0;

  for (;;) {
    if (tid == 0) {
      const u64 t = atomicAdd(a.task_ctr, 1ull);
      S.task = t;
      if (t < a.ntask) {
        u32 lo = 0, hi = a.nitems;
        while (hi - lo > 1) {
          const u32 mid = (lo + hi) >> 1;
          if (a.task_prefix[mid] <= t) lo = mid; else hi = mid;
        }
        S.item = lo;
      }
    }
    __syncthreads();
    const u64 task = S.task;
    if (task >= a.ntask) break;
    const u32 gitem = a.item_index[S.item];
    const DevItem it = a.items[gitem];
    const u32 eidx = it.engine;
    const DevEngine& eg = a.engines[eidx];
    if (S.eng != eidx) {
      if (!stage_patterns<pat_bytes<P0, NS>()>(spat, eg.pat, &S.mbar, &S.status,
                                               phase, a.ctr))
        return;
      for (u32 i = tid; i <= eg.sbits_words; i += kBlock)
        S.sbits[i] = i < eg.sbits_words ? eg.sbits[i] : 0u;
      __syncthreads();
      if (tid == 0) S.eng = eidx;
    }
    const DevEngine e = eg;
    const u32* __restrict__ xq = a.xq + it.xq_off;
    const u32* __restrict__ kq = xq + mark_tests_at(e.nslots);
    const u64 tl = task - a.task_prefix[S.item];
    const u32 lane = (u32)(tl % e.L);
    const u64 chunk = tl / e.L;
    const u64 R = e.lanes[lane];
    const u64 u_start = chunk * (u64)SEG * a.seg_per_task;
    const u64 u_end = min((u64)it.U, u_start + (u64)SEG * a.seg_per_task);
    // the line offset of the task's first period: one scaled residue gives
    // each pattern prime's table index and each slot's first hit offset
    const u64 v0 = u_start * e.M + R;
    const u32 vl = (u32)v0 & ((1u << kRedcSplit) - 1u);
    const u32 vh = (u32)(v0 >> kRedcSplit);
    if (tid < NS) S.ph[tid] = redc_residue(load_rec(e.prec + tid), xq[tid], vl, vh);
    for (u32 s = e.slot0 + tid; s < e.nslots; s += kBlock)
      S.off16[s] = (unsigned short)redc_residue(
          load_rec(e.mrec + s), __ldg(xq + kNSMax + s), vl, vh);
    __syncthreads();
    for (u64 useg = u_start; useg < u_end; useg += SEG) {
      const u32 seg_len = (u32)min((u64)SEG, u_end - useg);
      // (a) the pattern words tid, tid + kBlock, ... (a warp whose words all
      // lie past the segment's end skips them: a short lane's last segment
      // leaves most warps idle)
      u64 acc[WPT];
#pragma unroll
      for (int k = 0; k < WPT; ++k) acc[k] = 0;
      if (64u * ((u32)tid & ~31u) < seg_len) {
        PatSeg<P0, 0, NS, WPT>::words(spat, S.ph, (u32)tid, acc);
        nword += WPT;
      }
      // zero the byte map up to the segment's end
      {
        uint4* b4 = reinterpret_cast<uint4*>(S.bytes);
        const uint4 z = make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int k = 0; k < SEG / 16 / kBlock; ++k) {
          const u32 idx = tid + k * kBlock;
          if (16u * idx < seg_len) b4[idx] = z;
        }
      }
      __syncthreads();
      // (b) mark
      nmark += seg_len == SEG
                   ? mark_segment<true, SEG>(S.bytes, S.off16, e, SEG)
                   : mark_segment<false, SEG>(S.bytes, S.off16, e, seg_len);
      __syncthreads();
      // advance the offsets and phases to the next segment (nothing below
      // reads them before the next segment's barrier)
      if (useg + SEG < u_end) {
        for (u32 s = e.slot0 + tid; s < e.nslots; s += kBlock) {
          const u32 m = __ldg(e.mq + s);
          const u32 q = m & 0xFFFFu;
          const u32 o = S.off16[s] + (m >> 16);
          S.off16[s] = (unsigned short)min(o, o - q);
        }
        if (tid < NS) {
          const PrimeRec pr = e.recs[tid];
          const u32 p = S.ph[tid] + (u32)(SEG / 64) % pr.q;
          S.ph[tid] = min(p, p - pr.q);
        }
      }
      // (c) extract
#pragma unroll
      for (int k = 0; k < WPT; ++k) {
        const u32 w = tid + k * kBlock;
        const u64 uw = useg + 64ull * w;
        if (uw >= u_end) continue;
        const u64 m = map_bits(S.bytes, w);
        const u64 left = u_end - uw;
        u64 valid = left >= 64 ? ~0ull : ((1ull << left) - 1ull);
        if (uw == 0 && R < it.lo_off) valid &= ~1ull;
        if (it.U - uw <= 64 && R >= it.hi_last)
          valid &= ~(1ull << (it.U - uw - 1));
        u64 surv = ~acc[k] & ~m & valid;
        while (surv) {
          const int b = __ffsll((long long)surv) - 1;
          surv &= surv - 1;
          const u64 v = (uw + b) * e.M + R;
          bool alive = true;
          if (e.NPm < e.NP) {
            switch (test_mode(e, e.NPm)) {
              case TEST_EULER:
              case TEST_EULER_LOW:
                alive = tail_alive<TEST_EULER_LOW>(v, e, kq, S.sbits, ntest); break;
              case TEST_DICKSON:
                alive = tail_alive<TEST_DICKSON>(v, e, kq, S.sbits, ntest); break;
              case TEST_AP:
                alive = tail_alive<TEST_AP>(v, e, kq, S.sbits, ntest); break;
              default:
                alive = tail_alive<TEST_AP_DIV>(v, e, kq, S.sbits, ntest); break;
            }
          }
          if (!alive) continue;
          const unsigned long long p = atomicAdd(&a.ctr->ncand, 1ull);
          if (p < a.cand_cap) {
            a.cand_key[p] = v;
            a.cand_item[p] = gitem;
          } else {
            atomicOr(&a.ctr->overflow, 1u);
          }
        }
      }
      __syncthreads();
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    nmark += __shfl_down_sync(0xffffffffu, nmark, o);
    ntest += __shfl_down_sync(0xffffffffu, ntest, o);
    nword += __shfl_down_sync(0xffffffffu, nword, o);
  }
  if ((tid & 31) == 0) {
    if (nmark) atomicAdd(&a.ctr->marks, (unsigned long long)nmark);
    if (ntest) atomicAdd(&a.ctr->s2_tests, (unsigned long long)ntest);
    if (nword) atomicAdd(&a.ctr->s1_words, (unsigned long long)nword);
  }
}

}  // namespace fk
