"""The marking sieve's slots, pairs and fixed hit sequences.

For each engine the stream of the marking sieve must be the rounds kernel's
(checked against the oracle in test_gpu_rounds.py): one residue per prime
and many, residue counts that differ between primes (Dickson), primes that
divide the difference, sieves that end inside an octave and past 2^16, lanes
shorter and longer than a segment, at every segment length, both low-prime
forms and bounds of the marked range inside a block.  Whole numbers: equal.
"""

import pytest

import fk_abi

pytestmark = pytest.mark.gpu

TUNINGS = [dict(), dict(mark_segment=16384, mark_pattern_primes=24),
           dict(mark_segment=65536, mark_pattern_primes=40),
           dict(mark_segment=65536, mark_pattern_primes=24, seg_per_task=3),
           dict(mark_segment=32768, mark_pattern_primes=32, mark_limit=5000,
                seg_per_task=1),
           dict(mark_limit=1000)]


@pytest.mark.parametrize("kind,n,q2,d,p0,span", [
    (fk_abi.EULER, 1, 65536, None, 6, 10 ** 8),
    (fk_abi.EULER, 3, 65536, None, 6, 3 * 10 ** 9),
    (fk_abi.EULER, 5, 5000, None, 7, 3 * 10 ** 9),
    (fk_abi.EULER, 60, 65536, None, 6, 10 ** 9),
    (fk_abi.DICKSON, 6, 65536, None, 6, 2 ** 30),
    (fk_abi.DICKSON, 3, 1 << 18, None, 7, 2 ** 28),
    (fk_abi.DICKSON, 9, 300, None, 9, 2 ** 28),
    (fk_abi.AP, 1, 65536, None, 6, 2 ** 28),
    (fk_abi.AP, 6, 65536, None, 7, 2 ** 33),
    (fk_abi.AP, 4, 1 << 17, 30030 * 1009 * 65519, 6, 2 ** 29),
])
def test_marks_equal_rounds(kind, n, q2, d, p0, span):
    lo = 10 ** 13 + 11
    want = fk_abi.Engine(kind, n, q2=q2, d=d, p0=p0,
                         sieve="rounds").sieve(lo, lo + span).tolist()
    e = fk_abi.Engine(kind, n, q2=q2, d=d, p0=p0, sieve="mark")
    for t in TUNINGS:
        e.set_tuning(**t)
        assert e.sieve(lo, lo + span).tolist() == want, t
        if e.use_mark:
            assert e.stats()["marks"] > 0
