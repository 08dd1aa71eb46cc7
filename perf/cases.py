"""The sweeps a user of this framework runs, as measured cases.

Every case goes through a public entry point: the reference-API engines
(``euler_gpu``, ``ladder_gpu``, ``ap_gpu``), the batched engine
(``fk_batch.BatchEngine``), its submit / wait form as the serving loop uses
it, and the plain per-interval engine (``fk_batch.PlainEngine``).  The sizes
are the repository's workloads (``fk_workloads``), its fingerprinted score
windows and its plain configurations, from sweeps of a million candidates to
windows of 2e16.

A case fixes the shape of the work (engine kinds, filter sizes, lengths,
sieve depth, range of the starts); the seed draws where on the line the
intervals start.  Results are whole numbers: per interval the number of hits,
and the ordered offsets from each interval's start with the chain depths,
copied into the state's own buffers (of one size for all seeds, zero past the
last hit).
"""

import functools
import math
import os
import sys

import numpy as np

_PKG = os.path.abspath("first-knowns_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

EULER, DICKSON, AP = 0, 1, 2


# ------------------------------------------------------------------ cases ---

def listed():
    return [
        # the whole line from its start: the dense low pass below the engine
        # floor, then one short sweep -- two small calls, all latency
        dict(name="euler_line_2e20", call="euler_sweep", n=5, length=2 ** 20,
             start_lo=0.5, start_hi=4.5),
        # one plain hunt of the p < 1e9 configuration's size
        dict(name="euler_hunt_1e9", call="euler_hunt", n=8, length=10 ** 9,
             start_lo=9.0, start_hi=11.0, cap=64),
        # the score windows of 5e14 (SCORE at 1e16, SCORE128 at 2.3e20):
        # the widest wheel, lanes of a few dozen words
        dict(name="euler_stream_5e14", call="euler_stream", n=17,
             length=5 * 10 ** 14, start_lo=16.0, start_hi=20.4),
        # the campaign window (SCORE_WIDE at 6.11e20): lanes of 1563 words,
        # the longest single call
        dict(name="euler_stream_2e16", call="euler_stream", n=17,
             length=2 * 10 ** 16, start_lo=20.3, start_hi=21.0),
        # k below 2^34 with the deep sieve (q2 = 2^20): the plain Dickson
        # configuration, 82,000 sieve primes
        dict(name="dickson_hunt_2e34", call="dickson_hunt", n=6,
             q2=1 << 20, length=2 ** 34, start_lo=8.0, start_hi=10.5),
        # the Dickson score window (SCORE13): 2^38 of the j line
        dict(name="dickson_stream_2e38", call="dickson_stream", n=13,
             q2=65536, length=2 ** 38, start_lo=16.5, start_hi=17.2),
        # a quarter of the 13#-difference line: chains of ten and more
        dict(name="ap_chains_2e38", call="ap_chains", n=10, d=30030,
             length=2 ** 38, start_lo=12.0, start_hi=12.3, depth=10, cap=16),
        # the AP score window, its survivors as the launcher reads them
        dict(name="ap_stream_1e10", call="ap_stream", n=16, q2=65536,
             length=16106127360, start_lo=13.5, start_hi=14.0),
        # the headline workload, a sixteenth of its 4096 intervals
        dict(name="mixed_batch_256", call="batch", count=256, shape=1,
             len_lo=20.0, len_hi=36.0, thr_lo=4, thr_hi=12, start_lo=10.0,
             start_hi=18.0),
        # many short intervals in one batch, where set-up per interval counts
        dict(name="mixed_batch_short", call="batch", count=512, shape=2,
             len_lo=20.0, len_hi=27.0, thr_lo=4, thr_hi=12, start_lo=10.0,
             start_hi=18.0),
        # one slot's turn in the serving loop: chunks of requests, values to
        # 160 bits, new intervals every time and no graph
        dict(name="served_64", call="served", count=64, shape=3, len_lo=16.0,
             len_hi=30.0, thr_lo=6, thr_hi=14, start_lo=18.0, start_hi=24.0),
        # the same engines one call per interval
        dict(name="plain_mixed_24", call="plain", count=24, shape=4,
             len_lo=20.0, len_hi=31.0, thr_lo=4, thr_hi=12, start_lo=10.0,
             start_hi=18.0),
    ]


def draw(rng):
    """One more case of the listed ones' ranges."""
    def size(lo, hi):
        return int(2.0 ** rng.uniform(lo, hi)) | 1

    call = rng.choice(["euler_sweep", "euler_hunt", "euler_stream",
                       "dickson_hunt", "dickson_stream", "ap_chains",
                       "ap_stream", "batch", "batch", "served", "plain"])
    if call == "euler_sweep":
        return dict(call=call, n=rng.randint(4, 6), length=size(20, 24),
                    start_lo=0.5, start_hi=4.5)
    if call == "euler_hunt":
        c = dict(call=call, n=rng.randint(4, 10), length=size(22, 36),
                 start_lo=9.0, start_hi=12.0, cap=rng.choice([64, 100]))
        return _with_hits(c)
    if call == "euler_stream":
        n = rng.randint(15, 17)
        return dict(call=call, n=n, length=size(47, 54), start_lo=16.0,
                    start_hi=21.0)
    if call == "dickson_hunt":
        c = dict(call=call, n=rng.randint(5, 8),
                 q2=rng.choice([65536, 1 << 18, 1 << 20]),
                 length=size(30, 36), start_lo=8.0, start_hi=12.0)
        return _with_hits(c)
    if call == "dickson_stream":
        return dict(call=call, n=rng.randint(10, 13), q2=65536,
                    length=size(30, 38), start_lo=11.8, start_hi=17.2)
    if call == "ap_chains":
        c = dict(call=call, n=10, d=30030, length=size(34, 38),
                 start_lo=12.0, start_hi=12.3, depth=rng.randint(7, 10),
                 cap=16)
        return _with_hits(c)
    if call == "ap_stream":
        n = rng.randint(12, 16)
        return dict(call=call, n=n, q2=rng.choice([8192, 65536]),
                    length=30 * size(26, 30), start_lo=13.5, start_hi=18.0)
    shape = rng.randrange(1 << 20)
    if call == "batch":
        hi = rng.uniform(24, 36)
        return dict(call=call, count=int(2 ** rng.uniform(4, 8)), shape=shape,
                    len_lo=20.0, len_hi=hi, thr_lo=4, thr_hi=12,
                    start_lo=10.0, start_hi=18.0)
    if call == "served":
        return dict(call=call, count=int(2 ** rng.uniform(4, 7)), shape=shape,
                    len_lo=16.0, len_hi=30.0, thr_lo=6,
                    thr_hi=rng.randint(8, 14), start_lo=18.0, start_hi=24.0)
    return dict(call="plain", count=rng.randint(8, 32), shape=shape,
                len_lo=20.0, len_hi=31.0, thr_lo=4, thr_hi=12, start_lo=10.0,
                start_hi=18.0)


def _with_hits(case):
    """A hunt that finds something: the filter loosened until ten hits are
    expected."""
    while case["n"] > 4 and _expected(case)[1] < 10:
        case["n"] -= 1
        if case.get("depth", 0) > case["n"]:
            case["depth"] = case["n"]
    return case


# -------------------------------------------------- densities of the path ---

@functools.lru_cache(maxsize=None)
def _primes(below):
    f = np.ones(below, dtype=bool)
    f[:2] = False
    for q in range(2, int(below ** 0.5) + 1):
        if f[q]:
            f[q * q::q] = False
    return np.flatnonzero(f)


def _dickson_w(n):
    w = 1
    for q in _primes(n + 2):
        w *= int(q)
    return w


def _primorial(n):
    d = 1
    for q in _primes(400)[:n]:
        d *= int(q)
    return d


@functools.lru_cache(maxsize=None)
def _kill_rates(kind, n, q2, d):
    """(primes, share of the line that each of them kills)."""
    q = _primes(q2)
    if kind == EULER:
        f = np.minimum(n, (q + 1) // 2)
    elif kind == AP:
        d = d or _primorial(n)
        f = np.array([1 if p in (2, 3, 5) or d % int(p) == 0
                      else min(n, int(p)) for p in q])
    else:
        w = _dickson_w(n)
        f = np.full(q.shape, n)
        for i, p in enumerate(q[:300]):
            p = int(p)
            if w % p == 0:
                f[i] = 0
                continue
            s = (w * np.arange(p, dtype=np.int64) % p) ** 2 % p
            dead = np.zeros(p, dtype=bool)
            for m in range(1, n + 1):
                dead |= (m * s + 1) % p == 0
            f[i] = int(dead.sum())
    return q, f / q


@functools.lru_cache(maxsize=None)
def _density(kind, n, q2, d):
    """Of one unit of the line: positions a wheel of 2 ... 31 leaves, prime
    tests past the first 38 primes until one kills, survivors."""
    q, r = _kill_rates(kind, n, q2, d)
    keep = np.cumprod(1.0 - r)
    return keep[10], float(keep[37:].sum()), float(keep[-1])


def _spec(kind, n, q2, d, units, value_log10, depth):
    """(integer operations, hits) of sweeping `units` of the line: one OR of
    64 positions per pattern prime, nine multiply-adds per prime test, and
    for a hunt (depth > 0) the squarings of the chains' strong tests; a value
    with no factor below q2 is prime with probability e^gamma ln q2 / ln v."""
    wheel, tests, surv = _density(kind, n, q2, d)
    ops = units * (wheel * 32 / 64 + tests * 9)
    left = units * surv
    if depth:
        bits = value_log10 * math.log2(10) * (2 if kind == DICKSON else 1)
        words = math.ceil(bits / 32)
        p = min(1.0, 1.781 * math.log(q2) / (bits * math.log(2)))
        ops += left / max(1 - p, 0.05) * bits * (4 * words ** 2 + 2 * words)
        left *= p ** depth
    return ops, left


def _intervals(case):
    """(kind, n, q2, d, length, depth) of each interval of a list case."""
    rng = np.random.default_rng(case["shape"])
    c = case["count"]
    kinds = rng.integers(0, 3, size=c).tolist()
    lens = np.exp2(rng.uniform(case["len_lo"], case["len_hi"], size=c))
    thr = rng.integers(case["thr_lo"], case["thr_hi"] + 1, size=c).tolist()
    return [(k, t, 65536, 0, max(30, int(x) - int(x) % 30 if k == AP
                                 else int(x)), t)
            for k, x, t in zip(kinds, lens, thr)]


def _single(case):
    kind = {"e": EULER, "d": DICKSON, "a": AP}[case["call"][0]]
    hunt = case["call"] in ("euler_sweep", "euler_hunt", "dickson_hunt",
                            "ap_chains")
    depth = case.get("depth", case["n"]) if hunt else 0
    return (kind, case["n"], case.get("q2", 65536), case.get("d", 0),
            case["length"], depth)


def _expected(case):
    """(integer operations, hits) over the whole case."""
    rows = _intervals(case) if "count" in case else [_single(case)]
    ops = hits = 0.0
    for kind, n, q2, d, length, depth in rows:
        units = length
        if kind == DICKSON and case["call"] != "dickson_stream":
            units = length / _dickson_w(n)
        # hits are densest where values are smallest
        value = max(case["start_lo"], math.log10(max(length, 10)) - 1)
        o, h = _spec(kind, n, q2, d, units, value, depth)
        ops += o
        hits += h
    return ops, hits


def work(case):
    ops, hits = _expected(case)
    rows = case.get("count", 1)
    return {"bytes": float(48 * rows + 9 * hits), "flops": float(ops)}


# ---------------------------------------------------------------- running ---

@functools.lru_cache(maxsize=None)
def _engines():
    """The resident device engines of a process (a serving program's set)."""
    from fk_batch import EngineSet
    return EngineSet()


@functools.lru_cache(maxsize=None)
def _slot():
    """One serving slot: its buffers outlive the requests."""
    from fk_batch import BatchEngine
    return BatchEngine(engset=_engines())


def _start(rng, case):
    return int(10.0 ** rng.uniform(case["start_lo"], case["start_hi"]))


def prepare(case, seed):
    import fk_workloads as W
    rng = np.random.default_rng([int(seed), 77])
    call = case["call"]
    rows = case.get("count", 1)
    cap = int(4 * _expected(case)[1]) + 32 * rows + 1024
    st = {"call": call, "case": case,
          "count": np.zeros(rows, dtype=np.int64),
          "offset": np.zeros(cap, dtype=np.int64),
          "depth": np.zeros(cap, dtype=np.uint8)}
    if "count" in case:
        ivs = []
        for kind, n, _q2, _d, length, thr in _intervals(case):
            lo = _start(rng, case)
            if kind == EULER:
                lo = min(lo, W.EULER_CEIL - length)
            if kind == AP:
                lo -= lo % 30
            ivs.append(W.Interval(kind, n, lo, lo + length, thr,
                                  W.default_cap(kind, n)))
        st["intervals"] = ivs
        from fk_batch import BatchEngine, PlainEngine
        if call == "batch":
            st["engine"] = BatchEngine(ivs, engset=_engines())
        elif call == "served":
            st["engine"] = _slot()
            for iv in ivs:
                _engines().get(_engines().key_for(iv))
        else:
            st["engine"] = PlainEngine(engset=_engines())
            for iv in ivs:
                _engines().get(_engines().key_for(iv))
        return st
    lo = _start(rng, case)
    if call.startswith("euler"):
        import euler_gpu
        st["lo"] = max(lo, 2 if call == "euler_sweep" else 100_000)
        st["engine"] = euler_gpu.GpuEngine(case["n"])
    elif call.startswith("dickson"):
        import ladder_gpu
        st["lo"] = lo
        st["engine"] = ladder_gpu.GpuEngine(case["n"], q2=case["q2"])
    else:
        import ap_gpu
        st["lo"] = lo - lo % 30
        st["engine"] = (ap_gpu.GpuEngine(case["n"], d=case["d"])
                        if call == "ap_chains"
                        else ap_gpu.GpuEngine(case["n"], case["q2"]))
    return st


def _store(st, i, at, offsets, depths=None):
    """One interval's stream into the state's buffers; where it ends."""
    k = len(offsets)
    end = at + k
    if end > st["offset"].size:
        raise RuntimeError(f"{end} hits: more than the buffers hold")
    st["count"][i] = k
    st["offset"][at:end] = offsets
    if depths is not None:
        st["depth"][at:end] = depths
    return end


def run(st):
    case, call, eng = st["case"], st["call"], st["engine"]
    at = 0
    if "intervals" in st:
        ivs = st["intervals"]
        if call == "served":
            eng.submit(ivs)
            rows = eng.wait_arrays()
        else:
            rows = eng.run_arrays(ivs)
        for i, (off, dep) in enumerate(rows):
            at = _store(st, i, at, off, dep)
    else:
        lo, n, length = st["lo"], case["n"], case["length"]
        if call == "euler_sweep":
            import euler_gpu
            hits = euler_gpu.sweep(lo, lo + length, n)
        elif call == "euler_hunt":
            hits = eng.hunt(lo, lo + length, cap=case["cap"])
        elif call == "dickson_hunt":
            hits = eng.hunt(lo, lo + length)
        elif call == "ap_chains":
            hits = eng.hunt_cap(lo, length, case["depth"], case["cap"])
        else:
            hits = None
        if hits is not None:
            at = _store(st, 0, at, [x - lo for x, _ in hits],
                        [d for _, d in hits])
        elif call == "euler_stream":
            ps = eng.survivors_pre_mr(lo, lo + length)
            at = _store(st, 0, at, [p - lo for p in ps])
        elif call == "dickson_stream":
            js = eng.survivors_j(lo, lo + length)
            at = _store(st, 0, at, js - np.uint64(lo))
        else:
            parts = list(eng.survivors(lo, length))
            offs = np.concatenate(parts) if parts else np.zeros(0, np.uint64)
            at = _store(st, 0, at, offs)
    st["offset"][at:] = 0
    st["depth"][at:] = 0
    return {"count": st["count"], "offset": st["offset"],
            "depth": st["depth"]}
