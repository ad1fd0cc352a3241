"""Page-locked host memory that runs and models keep."""

import numpy as np
import pytest

import bitstreamzoo_b200 as bz
from bitstreamzoo_b200 import tuner
from bitstreamzoo_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _page_locked_mib():
    """Page-locked host memory of this process: the driver maps it shared."""
    with open("/proc/self/status") as f:
        return next(int(line.split()[1]) for line in f if line.startswith("RssShmem:")) / 1024


def _make_ring(ctx):
    """The device's ring of copy buffers, made by the first large copy."""
    a = wl.random_words(np.random.default_rng(2), 64 << 19)
    ctx.run("input stream a\noutput stream o\no = ~a\n", 64 << 19, {"a": a}).stream("o")


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
    before = _page_locked_mib()
    r = run(trips)
    assert r.int("n") == trips and r.stats["n_vm_launches"] >= trips
    assert _page_locked_mib() - before < 20


def test_large_calls_of_the_cost_model_keep_no_page_locked_copy(ctx):
    """48 MiB of rows in, 6 MiB of predictions out."""
    n = 1_500_000
    m = tuner.CostModel(ctx, 8, hidden=8, layers=1, seed=3)
    x = np.random.default_rng(1).normal(0, 1, (n, 8)).astype(np.float32)
    _make_ring(ctx)
    few = m.raw_predict(x[:1000])
    before = _page_locked_mib()
    out = m.raw_predict(x)
    del x
    assert out.shape == (n,) and np.array_equal(out[:1000], few)
    assert _page_locked_mib() - before < 20


def test_a_long_program_takes_no_page_locked_memory_for_its_list(ctx):
    """400,000 instructions with control flow, 6 MiB, run from device memory."""
    body = "\n".join(f"x = x {'^' if i % 2 else '|'} {'ab'[i // 2 % 2]}" for i in range(400_000))
    src = f"input stream a\ninput stream b\noutput stream x\nx = a\nif (a) {{\n{body}\n}}\n"
    prog = ctx.compile(src)
    ins = {"a": np.full(4, 5, dtype=np.uint64), "b": np.full(4, 9, dtype=np.uint64)}
    _make_ring(ctx)
    before = _page_locked_mib()
    r = ctx.run(prog, 256, ins, mode=bz.MODE_VM)
    assert r.stats["n_vm_launches"] == 1
    want = 5
    for i in range(400_000):
        v = (5, 9)[i // 2 % 2]
        want = want ^ v if i % 2 else want | v
    assert int(r.stream("x")[3]) == want
    assert _page_locked_mib() - before < 3
