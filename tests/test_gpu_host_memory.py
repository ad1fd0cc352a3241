"""Page-locked host memory that runs and models keep."""

import os

import numpy as np
import pytest

import bitstreamzoo_b200 as bz
from bitstreamzoo_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _mapped_mib():
    with open(f"/proc/{os.getpid()}/statm") as f:
        return int(f.read().split()[0]) * os.sysconf("SC_PAGE_SIZE") / 2**20


def test_a_long_walk_on_a_short_stream_keeps_no_list_per_segment(ctx):
    """4,000 trips whose segment is some 900 instructions, 15 KiB: 60 MiB in
    all, of which no more than a few are in use."""
    ops, trips, words = 900, 4_000, 70
    steps = ["^ a", "| b", "^ m"]
    body = "\n".join(f"  stream u{i} = {'x' if i == 0 else f'u{i - 1}'} {steps[i % 3]}" for i in range(ops))
    src = ("input stream a\ninput stream b\ninput stream m\noutput stream x\noutput int n\nx = a\nn = 0\n"
           f"int trips = popcount(m)\nfor i in 0..trips {{\n{body}\n  stream v = u{ops - 1} & a\n  x = u{ops - 1}\n"
           "  if (v) {\n    n = n + 1\n  }\n}\n")
    prog = ctx.compile(src)
    rng = np.random.default_rng(2)
    nbits = 64 * words
    ins = {"a": wl.random_words(rng, nbits), "b": wl.random_words(rng, nbits)}

    def run(k):
        m = np.zeros(words, dtype=np.uint64)
        m[: k // 64] = np.uint64(2**64 - 1)
        m[k // 64] = np.uint64((1 << (k % 64)) - 1)
        return ctx.run(prog, nbits, ins | {"m": m}, mode=bz.MODE_VM)

    run(20)
    before = _mapped_mib()
    r = run(trips)
    assert r.int("n") == trips and r.stats["n_vm_launches"] >= trips
    assert _mapped_mib() - before < 20
