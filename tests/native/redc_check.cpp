// Host check of fk_redc.h: the scaled residue of 55-bit values against
// 128-bit remainders.  Reads "q a x0 v" lines (decimal, x0 below 2^64);
// exits 1 at the first difference, printing it.
#include <cstdio>

#include "../../first-knowns_b200/csrc/fk_redc.h"

int main() {
  unsigned q;
  unsigned long long a, x0, v, n = 0;
  while (std::scanf("%u %llu %llu %llu", &q, &a, &x0, &v) == 4) {
    const fk::TestRec t = fk::redc_rec(q, a);
    const uint32_t k = (uint32_t)((x0 % q) * (uint64_t)t.c1 % q);
    const uint32_t got =
        fk::redc_residue(t, k, (uint32_t)(v & ((1ull << fk::kRedcSplit) - 1)),
                         (uint32_t)(v >> fk::kRedcSplit));
    const uint32_t want =
        (uint32_t)(((unsigned __int128)x0 + v) % q * (a % q) % q);
    if (got != want) {
      std::printf("q %u a %llu x0 %llu v %llu: %u, not %u\n", q, a, x0, v, got,
                  want);
      return 1;
    }
    ++n;
  }
  std::printf("%llu ok\n", n);
  return 0;
}
