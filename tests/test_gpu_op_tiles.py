"""Shifts, basis bits and the nonzero test at the edges of their tiles: 256 words per warp,
2,048 per block, vectors of two words, single bits at every kind of place, and
sources that are not 16-byte aligned."""

import numpy as np
import pytest

from oracle import cwords

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 32, 33, 255, 256, 257, 2047, 2048, 2049, 4096 + 31, 70_001]
SHIFTS = [0, 1, 63, 64, 65, 2047, 2048, 64 * 256, 64 * 256 + 1, 64 * 2049 - 1, 64 * 70_001, 64 * 70_001 + 5]


def dev(a):
    return torch.from_numpy(a.view(np.int64).copy()).cuda()


@pytest.mark.parametrize("n", SIZES)
def test_shift_tiles(ctx, n):
    rng = np.random.default_rng(n)
    a = rng.integers(0, 2**64, size=n, dtype=np.uint64)
    nbits = 64 * n - 3
    a[-1] &= np.uint64((1 << 61) - 1)
    da, dd = dev(a), torch.empty(n, dtype=torch.int64, device="cuda")
    for k in SHIFTS:
        torch.cuda.synchronize()
        ctx.op("shl", dd.data_ptr(), da.data_ptr(), k, n, nbits)
        ctx.sync()
        assert np.array_equal(dd.cpu().numpy().view(np.uint64), cwords.shl(a, k, nbits)), ("shl", k)
        for tail in (0, 1):
            torch.cuda.synchronize()
            ctx.op("shr", dd.data_ptr(), da.data_ptr(), k, n, tail)
            ctx.sync()
            ref = np.empty_like(a)
            cwords.lib().o_shr(cwords._p(ref), cwords._p(a), k, n, tail)
            assert np.array_equal(dd.cpu().numpy().view(np.uint64), ref), ("shr", k, tail)


@pytest.mark.parametrize("n", SIZES + [1 << 22, (1 << 22) + 1])
@pytest.mark.parametrize("offset", [0, 1])
def test_nonzero_single_bits(ctx, n, offset):
    t = torch.zeros(n + offset, dtype=torch.int64, device="cuda")
    p = t.data_ptr() + 8 * offset
    torch.cuda.synchronize()
    assert not ctx.is_nonzero(p, n)
    for w in sorted({0, n // 2, max(0, n - 2), n - 1}):
        t[w + offset] = 1 << (w % 63)
        torch.cuda.synchronize()
        assert ctx.is_nonzero(p, n), w
        t[w + offset] = 0
    if offset:
        t[0] = 1
    torch.cuda.synchronize()
    assert not ctx.is_nonzero(p, n)


# bytes: four steps of 32 words per warp from 2^18 words on
@pytest.mark.parametrize("n", [(64 << 18) - 64, 64 << 18, (64 << 18) + 1, (64 << 18) + 64 * 33 + 5, (64 << 18) + 64 * 511])
@pytest.mark.parametrize("offset", [0, 5])
def test_basis_bits_long(ctx, n, offset):
    from bitstreamzoo_b200 import workloads as wl

    data = np.random.default_rng(n).integers(0, 256, size=n + offset, dtype=np.uint8)
    src = torch.from_numpy(data).cuda()
    nw = (n + 63) // 64
    out = torch.full((8, nw + 1), -1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    ctx.s2p(src.data_ptr() + offset, n, [out[i].data_ptr() for i in range(8)])
    ctx.sync()
    got = out.cpu().numpy().view(np.uint64)
    for i, exp in enumerate(wl.basis_bits(data[offset:])):
        assert np.array_equal(got[i, :nw], exp), i
    assert (got[:, nw] == np.uint64(2**64 - 1)).all()
