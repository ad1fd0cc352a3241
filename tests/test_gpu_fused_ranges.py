"""Fused kernels at lengths where a walker's range is a few words or steps, so
that almost every word sits next to a speculated start state: deep DAGs of
additions and 1- to 70-bit shifts, and carries that run for many words, in
every kernel form, against the word-level oracle."""

import numpy as np
import pytest

import bitstreamzoo_b200 as bz
from bitstreamzoo_b200 import workloads as wl
from oracle import cwords, pyoracle

pytestmark = pytest.mark.gpu

FORMS = [None, {"layout": 0, "warps": 8, "min_blocks": 2, "prefetch": 0},
         {"layout": 1, "warps": 8, "min_blocks": 1}, {"layout": 1, "warps": 4, "min_blocks": 1, "chunk_words": 8},
         {"layout": 2, "chunk_words": 4, "warps": 8, "min_blocks": 1}]

# words: one range, around one step, a few ranges, around the TMA form's
# smallest stream and where every resident walker has a short range
WORDS = [1, 31, 33, 1000, 9473, (1 << 16) - 1, (1 << 16) + 5, 300_001]


def _check(ctx, src, nbits, inputs):
    ref_out, ref_pops = cwords.run_straight_line(pyoracle.parse(src), nbits, inputs)
    mask = np.uint64((1 << (nbits % 64)) - 1) if nbits % 64 else np.uint64(2**64 - 1)
    for form in FORMS:
        r = ctx.run(src, nbits, inputs, mode=bz.MODE_FUSED, schedule=form)
        for name, words in ref_out.items():
            exp = words.copy()
            exp[-1] &= mask
            got = r.stream(name)
            assert np.array_equal(got, exp), (form, name, int(np.argmax(got != exp)), got.size)
        for name, v in ref_pops.items():
            assert r.int(name) == v, (form, name)


@pytest.mark.parametrize("words", WORDS)
@pytest.mark.parametrize("max_shift", [1, 2, 70])
def test_deep_dags(ctx, words, max_shift):
    nbits = 64 * words - 7 * (words % 3)
    src = wl.shaped_dag_src(120, words + max_shift, window=12, p_bit=0.4, p_shl=0.3, p_add=0.25,
                            max_shift=max_shift, n_inputs=3)
    rng = np.random.default_rng(words)
    _check(ctx, src, nbits, {f"b{i}": wl.random_words(rng, nbits) for i in range(3)})


@pytest.mark.parametrize("words", WORDS)
@pytest.mark.parametrize("run_bits", [40, 700, 50_000])
def test_long_propagate_runs(ctx, words, run_bits):
    """y = ~x over runs of about ``run_bits`` bits: an addition's carry is
    undecided through each of them."""
    nbits = 64 * words - 1
    rng = np.random.default_rng(words + run_bits)
    x = wl.random_words(rng, nbits)
    y = x ^ ~wl.sparse_bits(rng, nbits, 1 / run_bits)
    wl._mask_tail(y, nbits)
    src = ("input stream x\ninput stream y\noutput stream s\noutput stream u\noutput int n\n"
           "s = x + y\nstream t = s << 3\nstream v = t + x\nstream w = v << 1\nu = w ^ s\nn = popcount(u)\n")
    _check(ctx, src, nbits, {"x": x, "y": y})
