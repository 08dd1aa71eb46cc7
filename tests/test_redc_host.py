"""The per-candidate tests' residue arithmetic (csrc/fk_redc.h), on the CPU.

The header compiles as plain C++: its scaled residue (X0 + v) * a mod q is
compared with 128-bit remainders at the edges of its range -- the smallest
sieve primes, primes just below and above 2^16, the largest prime below
2^30, values to 2^55 - 1 -- and on seeded draws over all of it.
"""

import pathlib
import random
import subprocess

ROOT = pathlib.Path(__file__).resolve().parents[1]


def test_residue_equals_the_128_bit_remainder(tmp_path):
    exe = tmp_path / "redc_check"
    subprocess.run(["g++", "-O1", "-std=c++17", "-o", str(exe),
                    str(ROOT / "tests" / "native" / "redc_check.cpp")],
                   check=True)
    rng = random.Random(20261205)
    primes = [17, 19, 23, 37, 191, 4093, 65521, 65537, 821641, 1048573,
              536870909, 1073741789]
    rows = []
    for q in primes:
        vs = [0, 1, q - 1, q, 2 ** 31 - 1, 2 ** 31, 2 ** 32 - 1, 2 ** 32,
              2 ** 55 - 1, (2 ** 55 - 1) // q * q,
              (2 ** 24 - 1) << 31] + [rng.randrange(2 ** 55)
                                      for _ in range(400)]
        for v in vs:
            for a in (1, q - 1, rng.randrange(1, q)):
                for x0 in (0, 2 ** 64 - 1, rng.randrange(2 ** 64)):
                    rows.append(f"{q} {a} {x0} {v}")
    out = subprocess.run([str(exe)], input="\n".join(rows) + "\n", text=True,
                         capture_output=True)
    assert out.returncode == 0, out.stdout
    assert out.stdout.strip() == f"{len(rows)} ok"
