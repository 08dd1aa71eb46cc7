"""The two SPRP kernels against the one-thread chain of fk_depths.

hunt() finds the base-2 depth with 1 to 32 lanes per candidate, by how many
candidates there are, and shares the exact tests out over a warp's lanes;
fk_depths runs the same chain serially in one thread per value.  For each
engine kind the hunt of a window must be the pre-primality stream filtered
by fk_depths, at candidate counts from none to past the one-lane-per-
candidate form, at depth caps from 0 up.  Whole numbers: equal.
"""

import pytest

import fk_abi

pytestmark = pytest.mark.gpu

# 75776 lanes on 148 SMs: 32 lanes per candidate to 2368 candidates, then
# 16, 8, 4, 2, and one past 37888
COUNTS = [0, 1, 30, 2300, 2500, 6000, 12000, 30000, 80000]


def _window(eng, lo, count):
    """[lo, hi) with about `count` pre-primality survivors."""
    return lo, lo + (int(count / eng.survival) if count else 1)


def _check(eng, lo, hi, thr, cap, scale=1, add=0):
    off = eng.sieve(lo, hi)
    dep = eng.depths([(lo + int(o)) * scale for o in off], cap)
    want = [(int(o), int(d)) for o, d in zip(off, dep) if d >= thr]
    got_o, got_d = eng.hunt(lo, hi, thr, cap)
    assert list(zip(got_o.tolist(), got_d.tolist())) == want
    return len(off)


@pytest.mark.parametrize("count", COUNTS)
def test_euler_and_ap_at_every_lane_split(count):
    eu = fk_abi.Engine(fk_abi.EULER, 4)
    n = _check(eu, *_window(eu, 10 ** 14, count), 3, 9)
    assert not count or n > count // 2
    ap = fk_abi.Engine(fk_abi.AP, 5, d=30030)
    _check(ap, *_window(ap, 10 ** 13, count), 4, 12)


@pytest.mark.parametrize("jlo", [10 ** 5, 10 ** 9, 10 ** 14, 10 ** 18])
@pytest.mark.parametrize("two_pass", [False, True])
def test_dickson_from_two_to_six_words(jlo, two_pass):
    e = fk_abi.Engine(fk_abi.DICKSON, 4, q2=4096, two_pass=two_pass)
    for count in (40, 6000):
        lo, hi = _window(e, jlo, count)
        _check(e, lo, hi, 2, 12, scale=e.W)


@pytest.mark.parametrize("thr,cap", [(0, 0), (0, 1), (1, 1), (2, 2), (0, 60),
                                     (3, 250)])
def test_depth_limits(thr, cap):
    eu = fk_abi.Engine(fk_abi.EULER, 3)
    lo, hi = _window(eu, 10 ** 12, 300)
    if thr <= cap:
        _check(eu, lo, hi, thr, cap)
    ap = fk_abi.Engine(fk_abi.AP, 3)
    _check(ap, *_window(ap, 10 ** 12, 300), thr, cap)


def test_dense_low_pass_from_two():
    """Every p from 2 up: the values include the primes trial division
    answers for, at every base."""
    e = fk_abi.Engine(fk_abi.EULER, 2)
    off, dep = e.dense(2, 5000, 1, 100)
    want = [(p - 2, int(d)) for p, d in
            zip(range(2, 5000), e.depths(range(2, 5000), 100)) if d >= 1]
    assert list(zip(off.tolist(), dep.tolist())) == want
