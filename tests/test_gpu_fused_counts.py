"""More popcounts in one kernel of the warp form than one round of its shared
memory holds (16 KiB: 512 at 4 warps, 256 at 8, 128 at 16)."""

import numpy as np
import pytest

import bitstreamzoo_b200 as bz
from bitstreamzoo_b200 import workloads as wl

pytestmark = pytest.mark.gpu


# 385 counts at 16 warps are past 48 KiB too, what a kernel may take at all
@pytest.mark.parametrize("warps,counts", [(16, 128), (16, 385)])
def test_counts_of_several_rounds(ctx, warps, counts):
    nbits = 64 * 9000
    names = [f"n{k}" for k in range(counts)]
    src = "\n".join(["input stream a"] + [f"output int {n}" for n in names] +
                    [line for k, n in enumerate(names) for line in (f"stream s{k} = a << {k % 16 + 1}", f"{n} = popcount(s{k})")])
    a = wl.random_words(np.random.default_rng(counts), nbits)
    below = np.concatenate([[0], np.cumsum(np.unpackbits(a.view(np.uint8), bitorder="little"), dtype=np.int64)])
    r = ctx.run(src + "\n", nbits, {"a": a}, mode=bz.MODE_FUSED,
                schedule={"layout": 0, "warps": warps, "min_blocks": 1, "prefetch": 0})
    assert [r.int(n) for n in names] == [int(below[nbits - k % 16 - 1]) for k in range(counts)]
    assert r.stats["n_fused_launches"] == 1
