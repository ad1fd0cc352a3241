"""Popcounts and conditions that a fused segment's last kernel hands to the
host itself: every kernel form, grids of one wave and of several, more counts
than it hands over, many segments in one run, runs in flight together."""

import numpy as np
import pytest

import bitstreamzoo_b200 as bz
from bitstreamzoo_b200 import workloads as wl

pytestmark = pytest.mark.gpu

FORMS = [None, {"layout": 0, "warps": 4}, {"layout": 0, "warps": 8, "prefetch": 1, "min_blocks": 4},
         {"layout": 1, "warps": 4, "min_blocks": 1}, {"layout": 2, "chunk_words": 4, "warps": 8, "min_blocks": 1}]


def _count(words):
    return int(np.unpackbits(words.view(np.uint8)).sum())


# words: one CTA, one wave, several waves of the warp form
@pytest.mark.parametrize("words", [3, 70_001, 4_000_003])
@pytest.mark.parametrize("form", range(len(FORMS)))
def test_counts_of_runs_in_flight(ctx, words, form):
    nbits = 64 * words - 5
    prog = ctx.compile("input stream a\ninput stream b\noutput stream o\noutput int n\noutput int m\n"
                       "o = a ^ b\nn = popcount(o)\nstream s = a & b\nm = popcount(s)\n")
    rng = np.random.default_rng(words)
    ins = [{k: wl.random_words(rng, nbits) for k in "ab"} for _ in range(3)]
    runs = []
    for i in ins:
        r = prog.run(nbits, bz.MODE_FUSED)
        if FORMS[form] is not None:
            r.set_schedule(FORMS[form])
        for k, v in i.items():
            r.bind(k, v)
        r.launch()
        runs.append(r)
    for r, i in zip(runs, ins):
        r.wait()
        assert r.int("n") == _count(i["a"] ^ i["b"])
        assert r.int("m") == _count(i["a"] & i["b"])
        assert np.array_equal(r.stream("o"), i["a"] ^ i["b"])


# counts: the most that are handed over (with the flags behind them), more
@pytest.mark.parametrize("counts", [1, 125, 126, 127, 200])
def test_many_counts(ctx, counts):
    nbits = 64 * 9000
    src = "\n".join(["input stream a", "output int t", "t = 0"] +
                    [line for k in range(counts) for line in
                     (f"stream s{k} = a << {k % 61}", f"int n{k} = popcount(s{k})", f"t = t + n{k}")]) + "\n"
    a = wl.random_words(np.random.default_rng(counts), nbits)
    bits = np.unpackbits(a.view(np.uint8), bitorder="little")
    want = sum(int(bits[:nbits - k % 61].sum()) for k in range(counts))
    assert ctx.run(src, nbits, {"a": a}, mode=bz.MODE_FUSED).int("t") == want


# trips: below, at and past what one fill of the slots covers
@pytest.mark.parametrize("trips", [1, 90, 300])
def test_many_segments(ctx, trips):
    nbits = 64 * 9000
    a = np.zeros(9000, dtype=np.uint64)
    a[8999] = np.uint64(1) << np.uint64(63)
    a[0] = np.uint64(1)
    a[(64 * 9000 - trips) // 64] |= np.uint64(1) << np.uint64((64 * 9000 - trips) % 64)
    src = ("input stream a\noutput int n\noutput int total\nstream x = a & a\nn = 0\ntotal = 0\n"
           f"stream one = ONES << {64 * 9000 - 1}\nstream pend = x\nstream keep = x >> 1\nkeep = keep << 1\n"
           "pend = keep\n"
           "while (pend) {\n  stream y = pend << 1\n  pend = y\n  int c = popcount(y)\n  total = total + c\n"
           "  n = n + 1\n}\n")
    got = {m: ctx.run(src, nbits, {"a": a}, mode=m) for m in (bz.MODE_FUSED, bz.MODE_PLAIN)}
    assert got[bz.MODE_FUSED].int("n") == got[bz.MODE_PLAIN].int("n") == trips
    assert got[bz.MODE_FUSED].int("total") == got[bz.MODE_PLAIN].int("total")
