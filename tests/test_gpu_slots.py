"""Runs that flush at many conditions: node ids kept across a flush, popcount
slots past one chunk, flags of segments without popcounts, and what a loop
compiles and keeps."""

import numpy as np
import pytest

import bitstreamzoo_b200 as bz
from bitstreamzoo_b200 import workloads as wl
from oracle import pyoracle

pytestmark = pytest.mark.gpu

WORDS = 150


def _bits(n, words=None):
    """A stream with its first n bits set."""
    w = np.zeros(words or (n + 63) // 64, dtype=np.uint64)
    w[: n // 64] = np.uint64(2**64 - 1)
    if n % 64:
        w[n // 64] = np.uint64((1 << (n % 64)) - 1)
    return w


def _count(w):
    return int(np.unpackbits(w.view(np.uint8)).sum())


# Slots are read and handed out again after 61,440: a loop takes 8 a trip with
# generated kernels (2 popcounts, 2 conditions, 2 flags and a counter beside
# each condition's segment), 4 on the interpreter; `first` popcounts in front
# put the end of the chunk at each of them in turn.
@pytest.mark.parametrize("mode,per_trip,first", [(bz.MODE_FUSED, 8, k) for k in range(8)] +
                         [(bz.MODE_VM, 4, k) for k in range(4)])
def test_values_across_the_end_of_a_chunk_of_slots(ctx, mode, per_trip, first):
    trips = 61440 // per_trip + 20
    words = max(WORDS, (trips + 63) // 64)
    rng = np.random.default_rng(first)
    nbits = 64 * words
    a, b = wl.random_words(rng, nbits), wl.random_words(rng, nbits)
    lines = ["input stream a", "input stream b", "input stream m", "output stream acc", "output int total",
             "output int hits", "total = 0", "hits = 0", "acc = ZERO", "int trips = popcount(m)"]
    for k in range(first):
        lines += [f"stream q{k} = a << {k + 1}", f"int e{k} = popcount(q{k})", f"total = total + e{k}"]
    lines += ["for i in 0..trips {", "stream u = a ^ b", "int c = popcount(u)", "stream w = a & b",
              "int d = popcount(w)", "total = total + c", "total = total + d",
              "stream v = u & b", "if (v) {", "hits = hits + 1", "stream t = acc ^ w", "acc = t", "}",
              "stream z = u & w", "if (z) {", "hits = hits + 1000000", "}", "}"]
    r = ctx.run("\n".join(lines) + "\n", nbits, {"a": a, "b": b, "m": _bits(trips, words)}, mode=mode)
    bits = np.unpackbits(a.view(np.uint8), bitorder="little")
    want = sum(int(bits[:nbits - k - 1].sum()) for k in range(first)) + trips * (_count(a ^ b) + _count(a & b))
    assert r.int("total") == want
    assert r.int("hits") == trips
    assert np.array_equal(r.stream("acc"), a & b if trips % 2 else np.zeros_like(a))


@pytest.mark.parametrize("mode", [bz.MODE_PLAIN, bz.MODE_FUSED, bz.MODE_VM])
def test_operands_across_an_int_that_has_to_be_read(ctx, mode):
    """The shift amount and the element's index are counts: the left operand,
    not computed yet, is computed with them."""
    src = ("input stream a\ninput stream b\ninput stream k\noutput stream x\noutput stream y\noutput stream w\n"
           "stream e[8]\ne[3] = a\nstream p = a & b\nw = p ^ a\n"
           "stream u = a ^ b\nstream h = k << 1\nint c = popcount(h)\nx = u << c\n"
           "stream v = a | b\nstream g = k << 2\nint d = popcount(g)\ny = v & e[d]\n")
    nbits = 64 * WORDS - 7
    rng = np.random.default_rng(5)
    inputs = {n: int.from_bytes(wl.random_words(rng, nbits).tobytes(), "little") for n in "ab"} | {"k": 0b10011}
    want, _, _ = pyoracle.run_source(src, nbits, inputs, {}, {})
    r = ctx.run(src, nbits, inputs, mode=mode)
    for name in "xyw":
        assert r.stream_int(name) == want[name] & ((1 << nbits) - 1), name


def test_more_segments_without_popcounts_than_a_chunk_has_slots(ctx):
    """A condition on an input takes no slot, the segment computed for it two."""
    trips, words = 35_500, 600
    rng = np.random.default_rng(3)
    a, b = wl.random_words(rng, 64 * words), wl.random_words(rng, 64 * words)
    src = ("input stream a\ninput stream b\ninput stream m\noutput stream acc\noutput int n\nn = 0\nacc = b\n"
           "int trips = popcount(m)\nfor i in 0..trips {\n  stream t = acc ^ a\n  acc = t\n"
           "  if (a) {\n    n = n + 1\n  }\n}\n")
    r = ctx.run(src, 64 * words, {"a": a, "b": b, "m": _bits(trips, words)}, mode=bz.MODE_FUSED)
    assert r.int("n") == trips
    assert np.array_equal(r.stream("acc"), b if trips % 2 == 0 else a ^ b)
    assert r.stats["n_fused_launches"] >= trips
