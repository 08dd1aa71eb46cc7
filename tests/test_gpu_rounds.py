"""The rounds kernel's per-candidate tests, at the edges of their forms.

Each case is one engine with the compaction rounds forced, its stream
compared with the CPU oracle's whole: weak filters (every pattern survivor
row fills the queues), Euler filters whose x^2 + x reach past the first
tested primes, differences that tested primes divide, sieves that end
inside the staged primes and sieves past 2^16, at each pattern-prime count
and with rounds on, off (warp_queue 513) and always (1).  Whole numbers:
equal, no tolerance.
"""

import pytest

import fk_abi
from oracle import ap as oap
from oracle import dickson as odk
from oracle import euler as oeu

pytestmark = pytest.mark.gpu

TUNINGS = [dict(), dict(pattern_primes=24, warp_queue=513),
           dict(pattern_primes=40, warp_queue=1, group_lane_words=8,
                warp_lane_words=64)]


def _check(eng, lo, hi, want):
    for t in TUNINGS:
        eng.set_tuning(**t)
        assert eng.sieve(lo, hi).tolist() == want, t


@pytest.mark.parametrize("n,p0,span", [(2, 6, 3 * 10 ** 6),
                                       (17, 6, 4 * 10 ** 9),
                                       (24, 6, 10 ** 10),
                                       (9, 9, 3 * 10 ** 8)])
def test_euler(n, p0, span):
    lo = 10 ** 12 + 12345
    want = [p - lo for p in oeu.CpuEngine(n).survivors_pre_mr(lo, lo + span)]
    _check(fk_abi.Engine(fk_abi.EULER, n, p0=p0, sieve="rounds"), lo,
           lo + span, want)


@pytest.mark.parametrize("n,q2,span", [(1, 65536, 200_000),
                                       (6, 600, 2 ** 20),
                                       (6, 1 << 18, 2 ** 20),
                                       (12, 65536, 2 ** 24)])
def test_dickson(n, q2, span):
    lo = 10 ** 11 + 77
    want = [int(j) - lo
            for j in odk.CpuEngine(n, q2=q2).survivors_j(lo, lo + span)]
    _check(fk_abi.Engine(fk_abi.DICKSON, n, q2=q2, sieve="rounds"), lo,
           lo + span, want)


@pytest.mark.parametrize("n,q2,d", [(2, 65536, None), (10, 257, None),
                                    (7, 1 << 17, 30030 * 1009 * 65537),
                                    (5, 65536, 30 * 211 * 40009),
                                    (9, 65536, 30030)])
def test_ap(n, q2, d):
    lo, span = 4 * 10 ** 13 - (4 * 10 ** 13) % 30, 30 * 2 ** 18
    ref = oap.CpuEngine(n, q2) if d is None else oap.CpuEngine(n, q2, d=d)
    want = ref.survivors(lo, span).tolist()
    _check(fk_abi.Engine(fk_abi.AP, n, q2=q2, d=d, sieve="rounds"), lo,
           lo + span, want)


def test_the_shared_out_rest_with_mixed_engines_and_a_full_list():
    """Candidates left in the warps' queues go to one list over all items of
    a batch: engines of every kind and depth side by side, in numbers that
    leave the list nearly empty and that overflow it (131072 entries; 256
    items leave up to 8 warps' queues on every CTA that joins them)."""
    engs = [fk_abi.Engine(fk_abi.EULER, 7, sieve="rounds"),
            fk_abi.Engine(fk_abi.DICKSON, 5, q2=1 << 18, sieve="rounds"),
            fk_abi.Engine(fk_abi.AP, 6, q2=300, sieve="rounds"),
            fk_abi.Engine(fk_abi.AP, 5, q2=1 << 17, sieve="rounds"),
            fk_abi.Engine(fk_abi.EULER, 3, sieve="rounds")]
    batch = fk_abi.Batch(engs)
    for items, span in ((5, 3000), (256, 3 * 10 ** 7)):
        specs = []
        for i in range(items):
            k = i % len(engs)
            lo = 10 ** 12 + i * 10 ** 9
            specs.append((k, fk_abi.MODE_SIEVE, 0, 0, lo,
                          lo + (span // 100 if k == 1 else span)))
        for graph in (False, True):
            rows = batch.run(specs, graph=graph)
            for (k, _m, _t, _c, lo, hi), (off, _d) in list(
                    zip(specs, rows))[::7 if items > 9 else 1]:
                assert off.tolist() == engs[k].sieve(lo, hi).tolist()
