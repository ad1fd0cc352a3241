"""The device interpreter gives a program back to the host past 2^27
instructions executed: what a condition skips is not executed."""

import numpy as np
import pytest

import bitstreamzoo_b200 as bz

pytestmark = pytest.mark.gpu


def test_skipped_instructions_do_not_count(ctx):
    """9,984 trips over a body of 14,000 instructions (1.4e8) behind a
    condition that is never met."""
    words = 156
    body = "\n".join("x = x ^ a" for _ in range(14_000))
    src = ("input stream a\ninput stream z\noutput stream x\noutput int n\nx = a\nn = 0\nstream t = a\n"
           f"while (t) {{\nif (z) {{\n{body}\n}}\nstream s = t << 1\nt = s\nn = n + 1\n}}\n")
    a = np.zeros(words, dtype=np.uint64)
    a[0] = np.uint64(1)
    r = ctx.run(src, 64 * words, {"a": a, "z": np.zeros_like(a)}, mode=bz.MODE_VM)
    assert r.int("n") == 64 * words
    assert np.array_equal(r.stream("x"), a)
    assert r.stats["n_vm_launches"] == 1
    assert r.stats["op_count"] == 64 * words
