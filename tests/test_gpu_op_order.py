"""Kernels launched while the one in front of them still runs: chains of
per-operator calls, each reading what the call before wrote, with nothing
between them, called directly and replayed from a captured graph; outputs that
are constants in runs on short streams."""

import numpy as np
import pytest

import bitstreamzoo_b200 as bz
from oracle import cwords

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(a.view(np.int64).copy()).cuda()


def _chain(ctx, x, y, z, n, nbits, rounds):
    for _ in range(rounds):
        ctx.op("xor", z.data_ptr(), x.data_ptr(), y.data_ptr(), n)
        ctx.op("shl", x.data_ptr(), z.data_ptr(), 65, n, nbits)
        ctx.op("add", y.data_ptr(), x.data_ptr(), z.data_ptr(), n, nbits)
        ctx.op("andnot", z.data_ptr(), y.data_ptr(), x.data_ptr(), n)
        ctx.op("not", x.data_ptr(), z.data_ptr(), n, nbits)
        ctx.op("or", z.data_ptr(), x.data_ptr(), y.data_ptr(), n)
        ctx.op("shr", y.data_ptr(), z.data_ptr(), 3, n, 0)


def _oracle(x, y, n, nbits, rounds):
    mask = np.full(n, 2**64 - 1, dtype=np.uint64)
    mask[-1] = np.uint64((1 << (nbits - 64 * (n - 1))) - 1)
    for _ in range(rounds):
        z = x ^ y
        x = cwords.shl(z, 65, nbits)
        y = cwords.add(x, z, nbits)
        z = y & ~x
        x = ~z & mask
        z = x | y
        y = np.empty_like(z)
        cwords.lib().o_shr(cwords._p(y), cwords._p(z), 3, n, 0)
    return x, y


# words: one block, one wave, several waves
@pytest.mark.parametrize("n", [5, 2049, 300_001, 3_000_001])
@pytest.mark.parametrize("captured", [False, True])
def test_chains(ctx, n, captured):
    nbits = 64 * n - 9
    rng = np.random.default_rng(n)
    hx, hy = (rng.integers(0, 2**64, size=n, dtype=np.uint64) for _ in range(2))
    for h in (hx, hy):
        h[-1] &= np.uint64((1 << 55) - 1)
    x, y, z = dev(hx), dev(hy), dev(hx)
    torch.cuda.synchronize()
    _chain(ctx, x, y, z, n, nbits, 1)   # the carry scan's scratch is there
    ctx.sync()
    x.copy_(dev(hx))
    y.copy_(dev(hy))
    torch.cuda.synchronize()
    if captured:
        s = torch.cuda.ExternalStream(ctx.stream)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            _chain(ctx, x, y, z, n, nbits, 2)
        with torch.cuda.stream(s):
            g.replay()
            g.replay()
    else:
        _chain(ctx, x, y, z, n, nbits, 4)
    ctx.sync()
    torch.cuda.synchronize()
    ex, ey = _oracle(hx, hy, n, nbits, 4)
    assert np.array_equal(x.cpu().numpy().view(np.uint64), ex)
    assert np.array_equal(y.cpu().numpy().view(np.uint64), ey)
    assert ctx.popcount(x.data_ptr(), n) == int(np.unpackbits(ex.view(np.uint8)).sum())


# words: one, the longest that stays in host memory, the first that does not
@pytest.mark.parametrize("words", [1, 8192, 8193])
@pytest.mark.parametrize("mode", [bz.MODE_AUTO, bz.MODE_VM, bz.MODE_PLAIN])
def test_constant_outputs(ctx, words, mode):
    nbits = 64 * words - 5
    src = ("input stream a\noutput stream o\noutput stream z\noutput stream k\noutput stream n\n"
           "o = a & a\nz = ZERO\nk = ONES\nn = ~z\n")
    a = np.random.default_rng(words).integers(0, 2**64, size=words, dtype=np.uint64)
    a[-1] &= np.uint64((1 << 59) - 1)
    ones = np.full(words, 2**64 - 1, dtype=np.uint64)
    ones[-1] = np.uint64((1 << 59) - 1)
    r = ctx.run(src, nbits, {"a": a}, mode=mode)
    want = {"o": a, "z": np.zeros_like(a), "k": ones, "n": ones}
    for name, exp in want.items():
        assert np.array_equal(r.stream(name), exp), name

        class View:
            __cuda_array_interface__ = {"shape": (words,), "typestr": "<i8", "version": 3, "strides": None,
                                        "data": (r.stream_device_ptr(name), False)}

        got = torch.as_tensor(View(), device="cuda").cpu().numpy().view(np.uint64).copy()
        got[-1] &= np.uint64((1 << 59) - 1)
        assert np.array_equal(got, exp), name
