"""Short streams that stay in page-locked host memory (inputs read, outputs
and popcounts written in place by the device interpreter), and conditions on
long streams whose counts come back with the speculation flags."""

import numpy as np
import pytest

import bitstreamzoo_b200 as bz
from bitstreamzoo_b200 import workloads as wl

pytestmark = pytest.mark.gpu

SRC = ("input stream a\ninput stream b\noutput stream same\noutput stream s\noutput stream z\noutput int n\noutput int m\n"
       "same = a\ns = a + b\nstream t = s << 65\nz = t ^ b\nn = popcount(z)\nm = popcount(s)\n")


def _ins(nbits, seed):
    rng = np.random.default_rng(seed)
    return {k: wl.random_words(rng, nbits) for k in "ab"}


# words: one, around a CTA, the longest in place, the first one copied
@pytest.mark.parametrize("words", [1, 47, 1024, 1025, 8192, 8193])
@pytest.mark.parametrize("mode", [bz.MODE_AUTO, bz.MODE_VM])
def test_overlapping_runs_and_reads(ctx, words, mode):
    """Runs launched one after the other before any is waited on, each with
    its own host inputs, overwritten by the caller right after binding."""
    torch = pytest.importorskip("torch")
    nbits = 64 * words - 3
    prog = ctx.compile(SRC)
    want, runs = [], []
    for k in range(6):
        ins = _ins(nbits, 100 * words + k)
        want.append(ctx.run(prog, nbits, ins, mode=bz.MODE_PLAIN))
        r = prog.run(nbits, mode)
        for name, v in ins.items():
            w = v.copy()
            r.bind(name, w)
            w[:] = 0
        r.launch()
        runs.append(r)
    for r, w in zip(runs, want):
        r.wait()
        for name in ("same", "s", "z"):
            exp = w.stream(name)
            assert np.array_equal(r.stream(name), exp), name

            class View:
                __cuda_array_interface__ = {"shape": (r.nw,), "typestr": "<i8", "version": 3, "strides": None,
                                            "data": (r.stream_device_ptr(name), False)}

            got = torch.as_tensor(View(), device="cuda").cpu().numpy().view(np.uint64).copy()
            got[-1] &= np.uint64((1 << 61) - 1)
            assert np.array_equal(got, exp), name
        assert (r.int("n"), r.int("m")) == (w.int("n"), w.int("m"))


def test_value_file_past_shared_memory_has_no_stale_host_copy(ctx):
    """More inputs than the value file holds: outputs come from the device."""
    n, nbits = 400, 64 * 6000 - 1
    src = "\n".join([f"input stream x[{n}]", "output stream o", "stream acc = ZERO", f"for i in 0..{n} {{",
                     "  stream t = acc ^ x[i]", "  acc = t", "}", "o = acc"]) + "\n"
    rng = np.random.default_rng(3)
    arrays = {"x": {i: wl.random_words(rng, nbits) for i in range(n)}}
    exp = np.zeros(6000, dtype=np.uint64)
    for v in arrays["x"].values():
        exp ^= v
    for mode in (bz.MODE_AUTO, bz.MODE_VM):
        r = ctx.run(src, nbits, input_arrays=arrays, mode=mode)
        assert np.array_equal(r.stream("o"), exp), mode


COND = """input stream a
input stream b
output stream acc
output int n
output int k
stream x = a & b
acc = x
n = popcount(x)
stream pend = x
while (pend) {
  stream adv = pend << 1
  stream w = adv & b
  stream y = w + b
  stream q = y ^ b
  stream got = q | adv
  stream na = ~acc
  stream fresh = got & na
  pend = fresh
  stream t = acc | got
  acc = t
  int step = popcount(fresh)
  n = n + step
}
stream none = x ^ x
if (none) {
  acc = a
}
if (a) {
  stream e = acc ^ a
  acc = e
}
k = popcount(acc)
"""


@pytest.mark.parametrize("nbits", [64 * 8193, (1 << 21) + 5])
@pytest.mark.parametrize("unproven", [False, True])
def test_conditions_on_long_streams(ctx, nbits, unproven):
    """unproven: operands whose carries never settle, so that conditions read
    counts of segments that are run again."""
    ins = _ins(nbits, nbits)
    ins["a"] &= wl.random_words(np.random.default_rng(1), nbits) & np.uint64(0x0101010101010101)
    src = COND
    if unproven:
        src = src.replace("stream x = a & b\n", "stream ia = ~a\nstream c = a + ia\nstream c2 = c << 1\n"
                          "stream c3 = c2 + a\nstream c4 = c3 & a\nstream x = c4 & b\n")
    want = ctx.run(src, nbits, ins, mode=bz.MODE_PLAIN)
    for mode in (bz.MODE_FUSED, bz.MODE_AUTO):
        r = ctx.run(src, nbits, ins, mode=mode)
        assert np.array_equal(r.stream("acc"), want.stream("acc")), mode
        assert (r.int("n"), r.int("k")) == (want.int("n"), want.int("k")), mode
        assert r.stats["op_count"] == want.stats["op_count"]


# words around the staged copies' 1 MiB chunk and 24-chunk ring
@pytest.mark.parametrize("words", [1 << 17, (1 << 17) + 1, 24 << 17, (24 << 17) + 1, (50 << 17) + 3])
def test_staged_copies(ctx, words):
    rng = np.random.default_rng(words)
    base = rng.integers(0, 2**64, size=words + 1, dtype=np.uint64)
    src = "input stream a\ninput stream b\noutput stream o\noutput stream p\no = a\np = a ^ b\n"
    a, b = base[1:], base[:-1]           # b: an address that is not 16-byte aligned with a's
    for _ in range(3):
        r = ctx.run(src, 64 * words, {"a": a, "b": b}, mode=bz.MODE_PLAIN)
        assert np.array_equal(r.stream("o"), a)
        assert np.array_equal(r.stream("p"), a ^ b)
