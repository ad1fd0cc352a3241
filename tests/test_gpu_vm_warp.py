"""Programs that the device interpreter runs in one warp (streams of up to 128
words), where lanes share words without a barrier of several warps between
them: a shift behind a popcount, ints that are their own operands."""

import numpy as np
import pytest

import bitstreamzoo_b200 as bz
from bitstreamzoo_b200 import workloads as wl

pytestmark = pytest.mark.gpu

# a value is written, counted (the int keeps the count on the device), shifted
SHIFT_AFTER_COUNT = """input stream a
input stream b
output stream acc
output int n
stream pend = a & a
acc = a
n = 0
while (pend) {
  stream s = acc ^ b
  int c = popcount(s)
  stream l = s << 1
  n = n + c
  stream u = l | b
  int d = popcount(u)
  stream r = u >> 1
  n = n - d
  acc = r
  stream p = pend << 97
  pend = p
}
"""

INTS = """input stream a
input stream b
output int n
output int m
output int k
output stream acc
stream z = a ^ b
n = popcount(z)
n = n + n
n = n * n
m = 0
k = 5
acc = b
stream pend = a
while (pend) {
  stream x = acc & pend
  int c = popcount(x)
  n = c - n
  m = m + c
  m = m * c
  k = k - m
  if (x) {
    k = c + k
    stream y = acc ^ pend
    acc = y
  }
  stream p = pend << 61
  pend = p
}
k = k - n
"""


@pytest.mark.parametrize("words", [1, 4, 5, 33, 127, 128])
@pytest.mark.parametrize("src", [SHIFT_AFTER_COUNT, INTS], ids=["shift", "ints"])
def test_one_warp(ctx, words, src):
    nbits = 64 * words - 3
    rng = np.random.default_rng(words)
    a = wl.random_words(rng, nbits)
    a[0] |= np.uint64(1)
    inputs = {"a": a, "b": wl.random_words(rng, nbits)}
    want = ctx.run(src, nbits, inputs, mode=bz.MODE_PLAIN)
    for _ in range(3):
        got = ctx.run(src, nbits, inputs, mode=bz.MODE_VM)
        assert got.stats["n_vm_launches"] == 1
        assert np.array_equal(got.stream("acc"), want.stream("acc"))
        for name in ("n", "m", "k")[:1 if src is SHIFT_AFTER_COUNT else 3]:
            assert got.int(name) == want.int(name), name
        assert got.stats["op_count"] == want.stats["op_count"]
