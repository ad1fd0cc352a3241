"""How far back a fused kernel proves its start states: carries that propagate
through thousands of words, which need no re-run by the per-op kernels."""

import numpy as np
import pytest

import bitstreamzoo_b200 as bz
from bitstreamzoo_b200 import workloads as wl
from oracle import cwords, pyoracle

pytestmark = pytest.mark.gpu

# enough arithmetic per stream for a thread form where no schedule is set
SRC = ("input stream x\ninput stream y\noutput stream o\noutput int n\n"
       "stream s = x + y\nstream t = s << 3\nstream v = t + x\nstream w = v << 1\no = w ^ s\nn = popcount(o)\n")
# shifts alone dirty 150 bits: a thread form's reach doubles
SHIFTS = ("input stream x\ninput stream y\noutput stream o\noutput int n\n"
          "stream a = x << 50\nstream b = a << 50\nstream c = b << 50\n"
          "stream s = x + y\no = s ^ c\nn = popcount(o)\n")


def _inputs(words, run):
    """y = ~x but for one bit in every ``run`` words: x + y propagates between them."""
    rng = np.random.default_rng(run)
    x = wl.random_words(rng, 64 * words)
    y = ~x
    y[run - 1::run] ^= np.uint64(1 << 17)
    return {"x": x, "y": y}


def _check(ctx, src, words, run, schedule, runs):
    ins = _inputs(words, run)
    ref, pops = cwords.run_straight_line(pyoracle.parse(src), 64 * words, ins)
    prog = ctx.compile(src)
    stats = []
    for _ in range(runs):
        r = ctx.run(prog, 64 * words, ins, mode=bz.MODE_FUSED, schedule=schedule)
        assert np.array_equal(r.stream("o"), ref["o"])
        assert r.int("n") == pops["n"]
        stats.append(r.stats)
    return stats


@pytest.mark.parametrize("src,schedule,run", [
    (SRC, {"layout": 0}, 12_000), (SRC, {"layout": 0, "warps": 8, "min_blocks": 2, "prefetch": 0}, 16_000),
    (SRC, {"layout": 1, "warps": 8, "min_blocks": 1}, 1_000),
    (SHIFTS, {"layout": 1, "warps": 4, "min_blocks": 1, "chunk_words": 8}, 1_900)])
def test_runs_within_reach(ctx, src, schedule, run):
    assert _check(ctx, src, 300_001, run, schedule, 1)[0]["n_fused_fallbacks"] == 0


@pytest.mark.parametrize("words", [70_001, 300_001])
@pytest.mark.parametrize("run", [6_000, 14_000])
def test_without_a_schedule_the_warp_form_takes_over(ctx, words, run):
    """The first run goes through both forms, the second starts in the warp form."""
    first, second = _check(ctx, SRC.replace("<< 3", f"<< {1 + run // 1000}"), words, run, None, 2)
    assert first["n_fused_fallbacks"] == second["n_fused_fallbacks"] == 0
    assert second["n_fused_launches"] == 1


def test_past_every_reach_the_result_is_exact(ctx):
    """A carry that never settles: both forms fail, then additions by look-back."""
    first, second = _check(ctx, SRC.replace("<< 3", "<< 29"), 70_001, 70_001, None, 2)
    assert first["n_fused_fallbacks"] >= 1
    assert second["n_fused_fallbacks"] == 0


def test_a_schedule_that_failed_does_not_decide_for_runs_without_one(ctx):
    """The schedule is the one that the executor picks at this length."""
    src = SRC.replace("<< 3", "<< 31")
    picked = {"layout": 1, "warps": 4, "min_blocks": 1, "prefetch": 0}
    assert _check(ctx, src, 70_001, 6_000, picked, 1)[0]["n_fused_fallbacks"] >= 1
    after = _check(ctx, src, 70_001, 6_000, None, 1)[0]
    assert after["n_fused_fallbacks"] == 0 and after["n_fused_launches"] == 1
