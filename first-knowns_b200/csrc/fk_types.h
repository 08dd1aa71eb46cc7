// fk_types.h -- device-side descriptors shared by host and kernels.
#pragma once
#include <cstdint>

#include "fk_redc.h"

namespace fk {

enum Kind : uint32_t { KIND_EULER = 0, KIND_DICKSON = 1, KIND_AP = 2 };

// How a prime's scaled residue is tested (fk_sieve.cuh): by kind, and for
// Euler and AP in a plain form without a branch and one for the primes that
// need more -- Euler's up to max(x^2 + x), and those that may divide d.
enum TestMode : uint32_t {
  TEST_EULER = 0, TEST_DICKSON = 1, TEST_AP = 2, TEST_EULER_LOW = 3,
  TEST_AP_DIV = 4,
};

// What an item asks for.
enum Mode : uint32_t {
  MODE_SIEVE = 0,   // pre-primality survivors only
  MODE_HUNT = 1,    // survivors classified; keep depth >= threshold
  MODE_DENSE = 2,   // no sieve: every x in the range is classified
};

// Per-prime record of the set-up work: base residues, lane shifts (16
// bytes).  The per-candidate tests have their own (TestRec, fk_redc.h).
struct PrimeRec {
  uint32_t q;
  uint32_t pad;
  uint64_t magic;   // floor(2^64 / q)
};

// Screen of a prime whose forbidden residues are an explicit list: bit
// (r & 31) of f0, (r >> 5 & 31) of f1 and (r >> 10 & 31) of f2 are set for
// every listed r, so a residue off the list passes all three only rarely;
// list = offset | count << 24 into the residue lists, in groups of four.
struct alignas(16) ListFilter {
  uint32_t f0, f1, f2, list;
};

constexpr int kBlock = 256;       // threads per CTA, every kernel
constexpr int kNS = 32;           // pattern primes per CTA (default)
constexpr int kNSMin = 24;        // fewest pattern primes a kernel variant
                                  // stages; marking tables start here
constexpr int kNSMax = 40;        // most: the engine's pattern tables hold
                                  // this many primes
constexpr uint32_t kPadWide = 64, kPadNarrow = 32;  // pattern table padding
constexpr int kMaxRounds = 64;
constexpr int kSortSmem = 4096;   // entries a CTA sorts in shared memory
constexpr int kClassChunk = 128;  // candidates a warp fetches at once
constexpr uint32_t kClassCtas = 2; // SPRP: CTAs an SM holds at their registers
constexpr int kSpecLanes = 512;   // SPRP: lanes an SM runs at no cost to each
constexpr int kBucketFill = 1024; // expected entries per ordering bucket
constexpr int kWarpMode = 32;     // warp queue below which a candidate
                                  // takes a whole warp
constexpr int kSbits = 512;       // Euler: most words of the {x^2 + x} bitset
constexpr int kStaged = 128;      // rounds: test primes held in shared memory
constexpr int kStagedBits = 1536; // Dickson: words of their residue bitmaps
constexpr int kRestCap = 1 << 17;  // rounds: candidates k_rest's list holds
constexpr int kMaxRun = 32;       // rounds: most blocks a warp claims at once
constexpr int kSeg = 32768;       // marking: periods per shared segment
                                  // (default; variants 16384 and 65536)
constexpr int kNumSeg = 3;        // marking segment variants
constexpr int kSegOf(int i) { return 16384 << i; }
constexpr int kSegPerTask = 8;    // marking: segments per task
constexpr int kMarkPrimes = 6528; // marking: most primes one engine marks,
                                  // counted from pattern prime kNSMin
                                  // (every prime from 7 to 2^16 fits)
constexpr int kMarkSlots = 7168;  // marking: most prime slots (the primes in
                                  // blocks of 32 by octave, each octave's
                                  // last block filled up)
constexpr int kMarkHits = 48;     // marking: hits per lane a pair item aims at
constexpr int kMarkCost = 800;    // marking: instructions a block item aims at

// One work item of the marking sieve, for one warp.  A lane's progressions
// are the f residues of its prime in each of nblk blocks of 32 slots, or,
// for the primes with many hits, one (slot, residue) pair of 32 of nearly
// equal step.  Marked are the hits hit0 ... hit0 + K - 1 of each (all of
// them inside a whole segment), then E more where they still lie inside it.
enum MarkKind : uint32_t {
  MARK_FIXED = 0,  // blocks, (K, E) one of (0, 1), (1, 1), (1 ... 7, 2);
                   // hit0 = 0
  MARK_BLOCKS = 1, // blocks, any K and E
  MARK_PAIRS = 2,
};
struct alignas(16) MarkItem {
  uint32_t kind;            // kind | nblk << 8 | f << 16
  uint32_t block;           // the first; pairs: their least prime
  uint32_t res;             // first word of the residue pairs, or of the pairs
  uint32_t hits;            // hit0 | K << 16 | E << 24
};

// Immutable per-engine tables (device-resident for the engine's life).
struct DevEngine {
  uint32_t kind, n, L, NP;        // NP: sieve primes (pattern + per-candidate)
  uint32_t P0, NS, nrounds, xxmax;  // NS: pattern primes of this batch's
                                    // kernel variant (kNSMin..kNSMax)
  uint32_t pat_words, sbits_words, two_pass, pad0;
  uint64_t M;                     // wheel period (x units)
  uint64_t W;                     // Dickson: k = W * j
  uint64_t d_lo, d_hi;            // AP difference
  const uint64_t* lanes;          // [L] admissible residues mod M, ascending
  // pattern words, compile-time layout: prime q's table holds q words,
  // entry k = the kill mask of the 64 periods from phase 64k mod q, so
  // consecutive words of a lane are consecutive entries
  const uint64_t* pat;
  // the rounds kernel's copies, every prime's table padded by kPadWide or
  // kPadNarrow entries that repeat its first ones
  const uint64_t* patw;
  const uint64_t* patn;
  const TestRec* prec;            // [kNSMax] pattern primes, a = 1 / (64 M):
                                  // the scaled residue of v = 64 M w + R is
                                  // the table index of word w of lane R
  const PrimeRec* recs;           // [NP]
  const uint32_t* c64;            // [NP] 2^64 mod q
  // per-candidate tests: the scaled residue r = (X0 + v) * a mod q
  // (fk_redc.h), a by kind -- Euler -1 (killed: r among the x^2 + x), AP
  // -1/d (killed: r < n; for the primes dividing d a = -1 and r = 0),
  // Dickson 1 (killed: min(r, q - r) on the prime's list)
  const TestRec* trec;            // [NP]
  const ListFilter* filt;         // Dickson [NP]; AP with ap_div [NP]: f0 =
                                  // 1 when q divides d
  const uint32_t* lists;          // explicit forbidden-residue lists
  // Dickson, the primes from index kNSMin that a drain can stage: exact
  // bitmaps of the killed min(r, q - r), prime i's at word boff[i - kNSMin]
  const uint32_t* boff;
  const uint32_t* bits;
  uint32_t deep;                  // rounds: first prime past which 128 primes
                                  // kill less than a quarter
  uint32_t ap_div;                // AP: a prime past the pattern divides d
  const uint32_t* rounds;         // [nrounds + 1] prime-index cuts
  const uint32_t* sbits;          // Euler: bitset of {x^2 + x : x < n}
  // marking sieve (long lanes): the primes past the pattern are marked in a
  // per-lane byte map, up to index NPm (q below qlim)
  uint32_t NPm, use_mark, qlim;
  // the marked primes sit in slots, 32 to a block: a block's primes are of
  // one octave and of (nearly) one residue count, a short list repeating its
  // last residue and a short block its last prime (a mark is idempotent)
  uint32_t nslots, slot0;         // the slots this batch marks: [slot0, nslots)
  const TestRec* mrec;            // [nslots] a = 1 / M: the scaled residue of
                                  // v = M u + R is the offset of the period u
                                  // in the prime's hits
  const uint32_t* sprime;         // [nslots] prime index
  const uint32_t* mres;           // per block, word (j / 2) * 32 + lane: the
                                  // lane's forbidden period residues j, j + 1
  const uint32_t* mpair;          // residue | slot << 16
  // tables of this batch's segment length SEG (one set per variant)
  const uint32_t* mq;             // [nslots] q | (SEG mod q) << 16
  const MarkItem* mwork;          // each warp's items one after the other
  const uint32_t* mwoff;          // [9] where each warp's begin, and the end
};

// One unit of work: a sub-range of one engine's line.
struct DevItem {
  uint32_t engine, mode, threshold, cap;
  uint64_t X0_lo, X0_hi;          // line base (a multiple of M for sieves)
  uint64_t U;                     // periods (sieve) or x count (dense)
  uint64_t lo_off;                // first valid x - X0 (in period 0)
  uint64_t hi_last;               // valid iff R < hi_last in period U-1
  uint32_t Tc;                    // words per chain (per thread)
  uint32_t lane_threads;          // threads sweeping one lane: 1, 8 or 32;
                                  // thread t of a group takes words t,
                                  // t + lane_threads, ... of its block
  uint64_t nchunk;                // chains per lane
  uint64_t ntask;                 // task count (rounds: blocks)
  uint64_t xq_off;                // this item's base-residue table
                                  // (base_residue, fk_sieve.cuh)
  uint32_t marked;                // 1: the marking kernel sweeps this item
  uint32_t run;                   // rounds: blocks a warp claims at once
  uint64_t nchunk_u;              // marking: u-chunks per lane
};

// Output entry before ordering: item index + (key << 8 | depth).
struct OutRec {
  uint64_t packed;
  uint32_t item;
  uint32_t pad;
};

struct DevCounters {
  unsigned long long ncand;       // candidates written
  unsigned long long nout;        // outputs written
  unsigned int overflow;          // bit 0 cand, bit 1 out, bit 2 timeout,
                                  // bit 3 value past 192 bits
  unsigned int pad;
  unsigned long long s1_words;    // pattern-sieve words processed
  unsigned long long s2_tests;    // per-candidate prime tests
  unsigned long long imad_alg;    // algorithmic IMADs of the SPRP stage
  unsigned long long sprp_values; // values strong-tested
  unsigned long long marks;       // marking-sieve byte marks
  unsigned long long class_next;  // SPRP stage: next candidate chunk
  unsigned long long nrest;       // candidates listed for k_rest
  unsigned long long nexact;      // candidates listed for the exact tests
  unsigned long long exact_next;  // exact tests: next candidate chunk
};

}  // namespace fk
