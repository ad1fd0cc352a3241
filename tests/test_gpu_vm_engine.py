"""The device interpreter's cluster engine at the sizes where its split of the
words changes: one warp, several warps, 1 to 16 CTAs (1,024 words a CTA), the
last stream that a cluster holds and the first one past it, with the value
file in shared and in global memory; straight-line segments against the
word-level oracle, whole programs with control flow against per-op runs."""

import numpy as np
import pytest

import bitstreamzoo_b200 as bz
from bitstreamzoo_b200 import workloads as wl
from oracle import cwords, pyoracle

pytestmark = pytest.mark.gpu

# words: around a thread's 4, a warp's 128, a CTA's 1,024 and a cluster's 16,384
WORDS = [1, 3, 4, 5, 127, 128, 129, 1021, 1024, 1025, 2048, 2049, 6250, 8192, 16384, 16385]

SRC = """input stream a
input stream b
input stream c
output stream s
output stream l1
output stream l63
output stream l64
output stream l70
output stream lf
output stream r1
output stream r64
output stream rf
output stream m
output int ns
output int nm
stream nb = ~b
stream t = a + b
s = t
l1 = t << 1
l63 = l1 << 63
l64 = l63 << 64
l70 = l64 << 4170
lf = a << 65600
r1 = t >> 1
r64 = r1 >> 64
rf = nb >> 65601
stream u = l1 + nb
stream v = u ^ c
stream w = v | l63
m = w + w
ns = popcount(s)
nm = popcount(m)
"""


def _inputs(nbits, seed):
    rng = np.random.default_rng(seed)
    a = wl.random_words(rng, nbits)
    b = ~wl.sparse_bits(rng, nbits, 1 / 4096)     # carries span many words
    wl._mask_tail(b, nbits)
    return {"a": a, "b": b, "c": wl.random_words(rng, nbits)}


def _wide_src(n):
    """n values live at once: a value file past the cluster's shared memory."""
    lines = ["input stream a", "input stream b", "input stream c", "output stream o", "output int k"]
    lines += [f"stream t{i} = a << {i + 1}" for i in range(n)]
    lines += ["stream x0 = b + c"] + [f"stream x{i + 1} = x{i} + t{i}" for i in range(n)]
    lines += [f"o = x{n}", "k = popcount(o)"]
    return "\n".join(lines) + "\n"


def _check(ctx, src, nbits, inputs):
    ref_out, ref_pops = cwords.run_straight_line(pyoracle.parse(src), nbits, inputs)
    r = ctx.run(src, nbits, inputs, mode=bz.MODE_VM)
    assert r.stats["n_vm_launches"] == 1
    mask = np.uint64((1 << (nbits % 64)) - 1) if nbits % 64 else np.uint64(2**64 - 1)
    for name, words in ref_out.items():
        exp = words.copy()
        exp[-1] &= mask
        got = r.stream(name)
        assert np.array_equal(got, exp), (name, int(np.argmax(got != exp)))
    for name, v in ref_pops.items():
        assert r.int(name) == v, name


@pytest.mark.parametrize("words", WORDS)
@pytest.mark.parametrize("cut", [0, 1, 63])
def test_segments(ctx, words, cut):
    nbits = 64 * words - cut
    _check(ctx, SRC, nbits, _inputs(nbits, words))


@pytest.mark.parametrize("words", [100, 1024, 3000, 8192])
@pytest.mark.parametrize("live", [30, 120, 700])
def test_value_file_in_shared_and_global_memory(ctx, words, live):
    nbits = 64 * words - 9
    _check(ctx, _wide_src(live), nbits, _inputs(nbits, words + live))


PROGRAM = """input stream a
input stream b
input stream c
output stream acc
output stream neg
output int n
output int k
stream x = a & c
stream z = ZERO
acc = x
n = 0
if (z) {
  acc = b
}
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
stream far = acc >> 4097
if (far) {
  stream back = far << 130
  stream e = back ^ c
  acc = e
}
neg = ONES
neg = neg >> 3
k = popcount(acc)
"""


@pytest.mark.parametrize("words", WORDS)
def test_programs_with_control_flow(ctx, words):
    nbits = 64 * words - 5
    ins = _inputs(nbits, 7 * words)
    ins["c"] &= np.uint64(0x0101010101010101)
    want = ctx.run(PROGRAM, nbits, ins, mode=bz.MODE_PLAIN)
    got = ctx.run(PROGRAM, nbits, ins, mode=bz.MODE_VM)
    assert got.stats["n_vm_launches"] == 1
    for name in ("acc", "neg"):
        assert np.array_equal(got.stream(name), want.stream(name)), name
    for name in ("n", "k"):
        assert got.int(name) == want.int(name), name
    assert got.stats["op_count"] == want.stats["op_count"]
