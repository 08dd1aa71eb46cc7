"""The rounds kernel's warp queues under the densest rows.

With the weakest filters nearly every row of a warp's columns fills 20 to 32
places of its queue, so columns are flushed several times a word and the
queue is drained in the middle of a flush.  One, eight and thirty-two threads
to a lane; each stream is, entry for entry, the CPU oracle's (AP, n = 2) or
the numbers without a prime factor below 2^16 (Euler, n = 1: a plain sieve).
"""

import numpy as np
import pytest

import fk_abi
from oracle import ap as oap
from oracle.primes import primes_below

pytestmark = pytest.mark.gpu

# threads per lane by lane length: the 13# wheel's lanes are 2, 10 and 34
# words of 64 periods in these spans
FORMS = [(30030 * 64 * 2 - 17, {}),
         (30030 * 64 * 10 + 4321, dict(group_lane_words=8)),
         (30030 * 64 * 34 + 11, dict(warp_lane_words=32))]


def _rough(lo, span):
    """Offsets of the numbers in [lo, lo + span) no prime below 2^16
    divides."""
    alive = np.ones(span, dtype=bool)
    for q in primes_below(65536):
        alive[(-lo) % int(q)::int(q)] = False
    return np.flatnonzero(alive).tolist()


@pytest.mark.parametrize("span,tuning", FORMS)
@pytest.mark.parametrize("kind", [fk_abi.EULER, fk_abi.AP])
def test_dense_rows(kind, span, tuning):
    lo = 10 ** 12 + 30 * 4115
    span -= span % 30
    if kind == fk_abi.EULER:
        eng = fk_abi.Engine(kind, 1, sieve="rounds")
        want = _rough(lo, span)
    else:
        eng = fk_abi.Engine(kind, 2, sieve="rounds")
        want = oap.CpuEngine(2, 65536).survivors(lo, span).tolist()
    for queue in (1, 32, 513):
        eng.set_tuning(warp_queue=queue, **tuning)
        assert eng.sieve(lo, lo + span).tolist() == want


def test_a_full_rest_list_against_the_marking_sieve():
    """256 items of five engines whose warps offer the list of shared-out
    candidates about ten times what it holds: every stream is the marking
    sieve's, which has no such list."""
    kinds = [(fk_abi.EULER, 7, 65536), (fk_abi.DICKSON, 5, 1 << 18),
             (fk_abi.AP, 6, 300), (fk_abi.AP, 5, 1 << 17),
             (fk_abi.EULER, 3, 65536)]
    engs = [fk_abi.Engine(k, n, q2=q2, sieve="rounds") for k, n, q2 in kinds]
    marks = [fk_abi.Engine(k, n, q2=q2, sieve="mark") for k, n, q2 in kinds]
    specs = []
    for i in range(256):
        k = i % len(kinds)
        lo = 10 ** 12 + i * 10 ** 9
        span = 3 * 10 ** 5 if k == 1 else 3 * 10 ** 7
        specs.append((k, fk_abi.MODE_SIEVE, 0, 0, lo, lo + span))
    rows = fk_abi.Batch(engs).run(specs, graph=False)
    for (k, _m, _t, _c, lo, hi), (off, _d) in zip(specs, rows):
        assert np.array_equal(off, marks[k].sieve(lo, hi))
