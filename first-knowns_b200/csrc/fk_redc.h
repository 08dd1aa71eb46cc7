// fk_redc.h -- the scaled residue of a 55-bit value modulo a 30-bit prime.
//
// Montgomery reduction (Montgomery 1985) of one 32-bit word: with qi =
// q^-1 mod 2^32, N - (N * qi mod 2^32) * q is divisible by 2^32, so
// (N >> 32) - hi((N * qi mod 2^32) * q) is N * 2^-32 modulo q.  The sieve
// wants (X0 + v) * a mod q for a fixed a per prime (the scale that turns
// each engine's forbidden residues into a short test); the 2^32 the
// reduction divides by is put into the constants instead, so the value
// needs no other reduction:
//   c1 = a * 2^32, c2 = a * 2^63, k = X0 * a * 2^32   (all mod q)
//   N  = lo31(v) * c1 + (v >> 31) * c2 + k
// v < 2^55 splits at bit 31: N < q * (2^31 + 2^24), so the difference
// above lies in (-q, q) and one conditional add ends in [0, q).
#pragma once
#include <cstdint>

#if defined(__CUDACC__)
#define FK_REDC_HD __host__ __device__ __forceinline__
#else
#define FK_REDC_HD inline
#endif

namespace fk {

// Per-prime constants of the test: one 16-byte load.
struct alignas(16) TestRec {
  uint32_t q, qi, c1, c2;
};

constexpr int kRedcSplit = 31;
constexpr int kRedcBits = 55;

// a for prime q -> its record (host side, at engine construction).
inline TestRec redc_rec(uint32_t q, uint64_t a) {
  TestRec t;
  t.q = q;
  uint32_t inv = q;  // q * q == 1 mod 8: correct to 3 bits, doubled 4 times
  for (int i = 0; i < 4; ++i) inv *= 2u - q * inv;
  t.qi = inv;
  a %= q;
  t.c1 = (uint32_t)((a << 32) % q);
  t.c2 = (uint32_t)((((uint64_t)t.c1) << kRedcSplit) % q);
  return t;
}

// (X0 + v) * a mod q, in [0, q): vl = v mod 2^31, vh = v >> 31, k = X0 * c1
// mod q.
FK_REDC_HD uint32_t redc_residue(const TestRec& t, uint32_t k, uint32_t vl,
                                 uint32_t vh) {
#if defined(__CUDA_ARCH__)
  // spelled out, the chain is two wide and two plain multiply-adds and three
  // adds: 10.6 instructions a test with its loop, 1.92e12 tests/s, against
  // 11.9 and 1.65e12 as the compiler schedules the lines below
  uint32_t r;
  asm("{\n\t.reg .u64 n;\n\t.reg .u32 lo, hi, m, h, s;\n\t"
      "cvt.u64.u32 n, %2;\n\t"
      "mad.wide.u32 n, %3, %5, n;\n\t"
      "mad.wide.u32 n, %4, %6, n;\n\t"
      "mov.b64 {lo, hi}, n;\n\t"
      "mul.lo.u32 m, lo, %7;\n\t"
      "mul.hi.u32 h, m, %1;\n\t"
      "sub.u32 hi, hi, h;\n\t"
      "add.u32 s, hi, %1;\n\t"
      "min.u32 %0, hi, s;\n\t}"
      : "=r"(r)
      : "r"(t.q), "r"(k), "r"(vl), "r"(vh), "r"(t.c1), "r"(t.c2), "r"(t.qi));
  return r;
#else
  uint64_t n = (uint64_t)vl * t.c1 + k;
  n += (uint64_t)vh * t.c2;
  const uint32_t m = (uint32_t)n * t.qi;
  const uint32_t h = (uint32_t)(((uint64_t)m * t.q) >> 32);
  const uint32_t r = (uint32_t)(n >> 32) - h;
  const uint32_t s = r + t.q;
  return r < s ? r : s;  // a negative difference wraps above its sum with q
#endif
}

}  // namespace fk
