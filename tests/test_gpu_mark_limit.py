"""The marking sieve's bound and its short segments.

mark_limit decides which primes are marked and which are tested one by one:
the stream stays the rounds kernel's at every bound, in lanes of one period
and of several segments, and a low bound leaves the work above it undone.
"""

import pytest

import fk_abi

pytestmark = pytest.mark.gpu

LIMITS = [130, 300, 2047, 2048, 4093, 20011, 65536]


@pytest.mark.parametrize("kind,n,q2,p0,lo,span", [
    (fk_abi.DICKSON, 4, 1 << 17, 9, 6091, 53),        # one period a lane
    (fk_abi.EULER, 3, 65536, 6, 10 ** 12, 30030 * 70),
    (fk_abi.AP, 5, 65600, 6, 3 * 10 ** 13, 30030 * 70001),
])
def test_every_bound_gives_the_same_stream(kind, n, q2, p0, lo, span):
    want = fk_abi.Engine(kind, n, q2=q2, p0=p0,
                         sieve="rounds").sieve(lo, lo + span).tolist()
    e = fk_abi.Engine(kind, n, q2=q2, p0=p0, sieve="mark")
    for seg in (16384, 32768, 65536):
        for ns in (24, 32, 40):
            for limit in LIMITS:
                e.set_tuning(mark_segment=seg, mark_pattern_primes=ns,
                             mark_limit=limit)
                assert e.sieve(lo, lo + span).tolist() == want, (seg, ns, limit)


def test_a_low_bound_skips_what_lies_above_it():
    """One-period lanes, no candidate left for the tests: marking below 300
    is a small part of marking below 2^16."""
    e = fk_abi.Engine(fk_abi.DICKSON, 4, q2=1 << 17, p0=9, sieve="mark")
    ms = {}
    for limit in (65536, 300):
        e.set_tuning(mark_segment=65536, mark_limit=limit)
        t = []
        for _ in range(5):
            e.sieve(6091, 6144)
            t.append(e.stats()["mark_ms"])
        ms[limit] = min(t)
    assert ms[300] < 0.5 * ms[65536], ms
