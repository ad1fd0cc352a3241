"""The automatic mode asks for the kernel that the segment will take: buffers
that are not 32-byte aligned take the warp form, and a kernel of another form
does not stand for it."""

import numpy as np
import pytest

import bitstreamzoo_b200 as bz
from bitstreamzoo_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("compiled_at,runs_at", [(0, 0), (8, 8), (0, 8), (8, 0)])
def test_auto_mode_with_borrowed_buffers(ctx, compiled_at, runs_at):
    torch = pytest.importorskip("torch")
    words = 1 << 16
    # a DAG that takes a thread form where it may; its own for every parameter
    src = wl.shaped_dag_src(100, 8100 + compiled_at + 100 * runs_at, window=12, p_bit=0.4, p_shl=0.3, p_add=0.2,
                            max_shift=40, n_inputs=3)
    prog = ctx.compile(src)
    rng = np.random.default_rng(1)
    ins = {f"b{i}": wl.random_words(rng, 64 * words) for i in range(3)}
    bufs = {k: torch.zeros(words + 4, dtype=torch.int64, device="cuda") for k in ins}

    def run(mode, offset):
        r = prog.run(64 * words, mode)
        for k, v in ins.items():
            b = bufs[k][offset // 8: offset // 8 + words]
            b.copy_(torch.from_numpy(v.view(np.int64)))
            torch.cuda.synchronize()
            r.bind(k, ("borrow", b.data_ptr(), words))
        r.execute()
        return r

    first = run(bz.MODE_FUSED, compiled_at)
    assert first.stats["n_fused_launches"] >= 1
    got = run(bz.MODE_AUTO, runs_at)
    assert got.stats["compile_ms"] == 0
    assert (got.stats["n_fused_launches"] >= 1) == (compiled_at == runs_at)
    for name in (f"o{j}" for j in range(4)):
        if first.has_stream(name):
            assert np.array_equal(got.stream(name), first.stream(name))
