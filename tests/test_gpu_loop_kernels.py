"""A loop over long streams compiles its body once, however many trips it makes."""

import numpy as np
import pytest

import bitstreamzoo_b200 as bz

pytestmark = pytest.mark.gpu

NBITS = 64 * 9000

# pend walks up from one bit until it leaves the stream, one trip per bit
WHILE = ("input stream a\noutput int n\noutput int total\noutput stream seen\nn = 0\ntotal = 0\n"
         "stream pend = a & a\nseen = a\nwhile (pend) {\n  stream y = pend << 1\n  pend = y\n"
         "  stream s = seen | y\n  seen = s\n  int c = popcount(y)\n  total = total + c\n  n = n + 1\n}\n")
# a condition on a value just computed, a popcount, and as many trips as m has bits
FOR = ("input stream a\ninput stream m\noutput int n\noutput int total\noutput stream seen\nn = 0\ntotal = 0\n"
       "seen = a\nint trips = popcount(m)\nfor i in 0..trips {\n  stream y = seen << 1\n  int c = popcount(y)\n"
       "  total = total + c\n  stream t = y & seen\n  if (t) {\n    n = n + 1000\n  }\n  seen = y\n  n = n + 1\n}\n")


def _one_bit(at):
    w = np.zeros(NBITS // 64, dtype=np.uint64)
    w[at // 64] = np.uint64(1 << (at % 64))
    return w


@pytest.mark.parametrize("src", [WHILE, FOR], ids=["while", "for"])
@pytest.mark.parametrize("schedule", [None, {"layout": 1, "warps": 4, "min_blocks": 1}], ids=["default", "threads"])
def test_more_trips_compile_nothing_new(ctx, src, schedule):
    prog = ctx.compile(src)
    for trips, bound in ((4, None), (50, 0)):
        inputs = {"a": _one_bit(NBITS - trips)}
        if src is FOR:
            inputs["m"] = np.zeros(NBITS // 64, dtype=np.uint64)
            inputs["m"][5] = np.uint64((1 << trips) - 1)
        r = ctx.run(prog, NBITS, inputs, mode=bz.MODE_FUSED, schedule=schedule)
        assert (r.int("n"), r.int("total")) == (trips, trips - 1)
        if bound is not None:
            assert r.stats["compile_ms"] == bound


@pytest.mark.parametrize("schedule", [{"layout": 0}, {"layout": 2, "chunk_words": 4, "warps": 8, "min_blocks": 1}],
                         ids=["warp", "tma"])
def test_a_restored_walk_compiles_nothing_new(ctx, schedule):
    """The second run restores the first one's walk, whose values have other
    numbers once dead ones are left out."""
    words = 1 << 16
    src = ("input stream a\ninput stream b\noutput stream o\noutput int n\nstream d = a | b\nstream e = d << 9\n"
           "stream s = a + b\nstream t = s << 2\nstream u = t ^ a\nstream g = u >> 5\no = g & s\nn = popcount(o)\n")
    prog = ctx.compile(src)
    rng = np.random.default_rng(4)
    ins = {k: rng.integers(0, 2**64, words, dtype=np.uint64) for k in "ab"}
    first = ctx.run(prog, 64 * words, ins, mode=bz.MODE_FUSED, schedule=schedule)
    second = ctx.run(prog, 64 * words, ins, mode=bz.MODE_FUSED, schedule=schedule)
    assert not first.stats["walk_replayed"] and second.stats["walk_replayed"]
    assert second.stats["compile_ms"] == 0
    assert np.array_equal(second.stream("o"), first.stream("o")) and second.int("n") == first.int("n")
