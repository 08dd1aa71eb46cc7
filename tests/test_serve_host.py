"""What the serving loop charges a chunk for, on the CPU."""

import types

import pytest

import fk_serve
import fk_workloads as W


def _slots(q2, first):
    """Slots the marking tables give the primes past the 24th from `first`
    on: blocks of 32, the next eight primes in one, the rest by octave."""
    flags = bytearray([1]) * q2
    primes = []
    for p in range(2, q2):
        if flags[p]:
            primes.append(p)
            flags[p * p::p] = bytes(len(range(p * p, q2, p)))
    marked = [p for p in primes[first + 24:] if p < 65536]
    octaves = {}
    for p in marked[8:]:
        octaves[p.bit_length()] = octaves.get(p.bit_length(), 0) + 1
    return len(marked[8:]), 32 + sum(-(-c // 32) * 32
                                     for c in octaves.values())


@pytest.mark.parametrize("q2", [600, 4099, 40000, 65536, 1 << 18])
@pytest.mark.parametrize("first", [6, 7, 11])
def test_a_marked_chunk_is_charged_its_slots(q2, first):
    loop = fk_serve.ServeLoop.__new__(fk_serve.ServeLoop)
    marked, slots = _slots(q2, first)
    eng = types.SimpleNamespace(survival=1e-9, W=1, NP=6542, use_mark=True,
                                marked_primes=marked)
    loop._engine = lambda iv: eng
    iv = W.Interval(W.EULER, 6, 10 ** 12, 10 ** 12 + 1000, 6, 64)
    with_marks = loop.footprint(iv)
    eng.use_mark = False
    rounds = loop.footprint(iv)
    # the table of a marked item: every sieve prime, 40 pattern primes, slots
    assert with_marks - rounds >= 4 * (40 + slots)
    assert with_marks - rounds <= 4 * (40 + slots) + 2048
    assert rounds >= 4 * eng.NP
