"""Captured graphs between runs of other sizes.

One batch, run eagerly and from graphs with item counts that make its
buffers grow at different times; every result is that of a batch which ran
nothing else.  Whole numbers: equal.
"""

import pytest

import fk_abi

pytestmark = pytest.mark.gpu


def _specs(count, length, at=10 ** 12):
    return [(0, fk_abi.MODE_HUNT, 3, 64, at + i * (1 << 33),
             at + i * (1 << 33) + length) for i in range(count)]


def _lists(rows):
    return [(o.tolist(), d.tolist()) for o, d in rows]


@pytest.mark.parametrize("counts", [(684, 690, 1000, 1024),
                                    (700, 750, 1000, 1030)])
def test_a_graph_after_eager_runs_that_grew_buffers(counts):
    eng = fk_abi.Engine(fk_abi.EULER, 8, sieve="rounds")
    first, second, graphed, grown = counts
    want = _lists(fk_abi.Batch([eng]).run(_specs(graphed, 1 << 24),
                                          graph=False))
    more = _lists(fk_abi.Batch([eng]).run(_specs(grown, 1 << 24, 10 ** 13),
                                          graph=False))
    assert sum(len(o) for o, _ in want) > 100
    b = fk_abi.Batch([eng])
    b.run(_specs(first, 1 << 32), graph=False)   # the largest output expected
    b.run(_specs(second, 1 << 24), graph=False)
    assert _lists(b.run(_specs(graphed, 1 << 24), graph=True)) == want
    assert _lists(b.run(_specs(grown, 1 << 24, 10 ** 13), graph=False)) == more
    for _ in range(3):
        assert _lists(b.run(_specs(graphed, 1 << 24), graph=True)) == want


def test_results_around_the_short_read_back():
    """Streams of 0 to 4097 entries, 2047 to 2049 among them, from one graph
    batch whose result grows and shrinks, against the plain call's."""
    eng = fk_abi.Engine(fk_abi.EULER, 2, sieve="rounds")
    ref = fk_abi.Engine(fk_abi.EULER, 2, sieve="mark")
    lo = 10 ** 12
    off = ref.sieve(lo, lo + (1 << 22)).tolist()
    assert len(off) > 4097
    b = fk_abi.Batch([eng])
    for n in (4097, 0, 2048, 2049, 2047, 1, 4096, 2048):
        hi = lo + (off[n - 1] + 1 if n else off[0])
        for graph in (True, True, False):
            (got, _), = b.run([(0, fk_abi.MODE_SIEVE, 0, 0, lo, hi)],
                              graph=graph)
            assert got.tolist() == off[:n]
        assert eng.sieve(lo, hi).tolist() == off[:n]
