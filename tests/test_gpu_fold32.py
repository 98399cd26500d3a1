"""Value products of b = 32 tiles: block rows of 1 to 97 tiles around the batch
of 32, tiles with few and with many non-empty rows around the line between the
two ways of dealing words out, rows that run through whole batches; and the
terms of fp32 products laid out beforehand on a graph of enough tiles.  Whole
numbers, so that the fp32 sums are exact in any order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(gbo, src, dst, n):
    key = np.unique(np.asarray(src, np.int64) * n + np.asarray(dst, np.int64))
    rowptr = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(key // n, minlength=n), out=rowptr[1:])
    return gbo.Csr(rowptr, (key % n).astype(np.int32), n, n)


def _check(gbo, orc, csr, b, rng):
    n = csr.nrows
    g, ref = gbo.Graph.from_csr(csr, b), orc.pack(csr.rowptr, csr.colind, n, n, b)
    dy = gbo.DeviceBuffer(4 * n)
    lab = rng.permutation(n).astype(np.int32)
    g.bmv_minselect(gbo.DeviceBuffer.from_numpy(lab), dy)
    assert np.array_equal(dy.to_numpy(np.int32, n), orc.bmv_minselect(ref, lab))
    g.bmv_minplus(gbo.DeviceBuffer.from_numpy(lab.astype(np.uint32)), dy)
    assert np.array_equal(dy.to_numpy(np.uint32, n), orc.bmv_minplus(ref, lab.astype(np.uint32)))
    x, scale = rng.integers(0, 8, n).astype(np.float32), rng.integers(1, 4, n).astype(np.float32)
    dx, ds = gbo.DeviceBuffer.from_numpy(x), gbo.DeviceBuffer.from_numpy(scale)
    row = np.repeat(np.arange(n), np.diff(csr.rowptr))
    for d, w in ((None, x), (ds, x * scale)):
        g.bmv_float(dx, dy, 2.0, d, 1.0)
        want = 2 * np.bincount(row, weights=w[csr.colind], minlength=n) + 1
        assert np.array_equal(dy.to_numpy(np.float32, n), want.astype(np.float32))


@pytest.mark.parametrize("words", [1, 6, 7, 32])
def test_batches(gbo, orc, gpu, words):
    rng = np.random.default_rng(words)
    lengths = [1, 2, 31, 32, 33, 63, 64, 65, 97]
    n = 32 * 100 - 5
    src, dst = [], []
    for R, tiles in enumerate(lengths):
        for t, J in enumerate(np.sort(rng.permutation(99)[:tiles])):
            # rows 3 and 30 in every tile as far as `words` goes, the others drawn
            rows = ([3, 30] + list(rng.permutation(32)))[: words if t % 5 else 1]
            for r in rows:
                cols = rng.permutation(32)[: 1 + int(rng.integers(0, 3)) * (t % 7 == 0)]
                src += [32 * R + r] * len(cols)
                dst += list(32 * J + cols)
    _check(gbo, orc, _csr(gbo, src, dst, n), 32, rng)


@pytest.mark.parametrize("b", [4, 32])
def test_terms_beforehand(gbo, orc, gpu, b):
    rng = np.random.default_rng(b)
    n = 20_003 if b == 4 else 70_001
    src, dst = rng.integers(0, n, 20 * n), rng.integers(0, n, 20 * n)
    if b == 4:
        src, dst = np.concatenate([src] + [rng.integers(0, n, 20 * n) for _ in range(3)]), \
            np.concatenate([dst] + [rng.integers(0, n, 20 * n) for _ in range(3)])
    csr = _csr(gbo, src, dst, n)
    assert gbo.Graph.from_csr(csr, b).info().nblocks >= max(1 << 20, 4 * n)
    _check(gbo, orc, csr, b, rng)


@pytest.mark.parametrize("b", [8, 16, 32, 64])
def test_terms_beforehand_on_a_skewed_graph(gbo, gpu, b):
    """A million tiles, 3.5 a column, and a hub row far past the others (b = 8:
    not laid out)."""
    rng = np.random.default_rng(b)
    n = 300_007
    src = np.concatenate([rng.integers(0, n, 1_150_000), np.full(n, 77)])
    dst = np.concatenate([rng.integers(0, n, 1_150_000), np.arange(n)])
    csr = _csr(gbo, src, dst, n)
    g = gbo.Graph.from_csr(csr, b)
    info = g.info()
    assert info.nblocks >= 1 << 20 and info.nblockcols * info.nblockrows > 12 * info.nblocks
    x, scale = rng.integers(0, 8, n).astype(np.float32), rng.integers(1, 4, n).astype(np.float32)
    row = np.repeat(np.arange(n), np.diff(csr.rowptr))
    want = (2 * np.bincount(row, weights=(x * scale)[csr.colind], minlength=n) + 1).astype(np.float32)
    dx, ds, dy = gbo.DeviceBuffer.from_numpy(x), gbo.DeviceBuffer.from_numpy(scale), gbo.DeviceBuffer(4 * n)
    for _ in range(2):
        g.bmv_float(dx, dy, 2.0, ds, 1.0)
        assert np.array_equal(dy.to_numpy(np.float32, n), want)
