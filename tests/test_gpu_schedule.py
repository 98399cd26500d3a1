"""Work items of graphs with few tiles and one long block row: just short of
being cut finer, just past it, and past the most tiles an item takes at all.
All products against the oracle; fp32 over small whole numbers, whose sums are
exact in fp32 in any order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FINE = 32  # tiles of an item where a graph's tiles are few


def _graph(gbo, b, tiles):
    """A block row of `tiles` tiles (its last row full, its first with a bit
    per tile) above a band of width 3."""
    n = b * tiles + b // 2 + 1
    band = np.arange(n)
    src = [band, band[1:], np.zeros(tiles, np.int64), np.full(b * tiles, b - 1)]
    dst = [band, band[1:] - 1, np.arange(tiles) * b + b // 3, np.arange(b * tiles)]
    src, dst = np.concatenate(src).astype(np.int64), np.concatenate(dst).astype(np.int64)
    key = np.unique(src * n + dst)
    rowptr = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(key // n, minlength=n), out=rowptr[1:])
    return gbo.Csr(rowptr, (key % n).astype(np.int32), n, n)


@pytest.mark.parametrize("b", [4, 8, 16, 32, 64])
@pytest.mark.parametrize("tiles", [4 * FINE, 4 * FINE + 1, None])
def test_products(gbo, orc, gpu, b, tiles):
    most = 8192 // b
    tiles = tiles or most + 1
    csr = _graph(gbo, b, tiles)
    n = csr.nrows
    g, ref = gbo.Graph.from_csr(csr, b), orc.pack(csr.rowptr, csr.colind, n, n, b)
    info = g.info()
    cut = -(-tiles // FINE) if tiles > 4 * FINE else -(-tiles // most)
    assert info.nitems == info.nblockrows - 1 + cut and info.nsplit_rows == (cut > 1)
    rng = np.random.default_rng(b + tiles)
    x = (rng.random(n) < 0.5).astype(np.int32)
    xw = orc.pack_vector(x, b)
    dx = gbo.DeviceBuffer.from_numpy(xw.astype(gbo.WORD_DTYPE[b]))
    dy = gbo.DeviceBuffer(4 * n)
    want = orc.bmv_count(ref, xw)
    g.bmv_count(dx, dy)
    assert np.array_equal(dy.to_numpy(np.int32, n), want)
    base = rng.integers(0, 5, n).astype(np.float32)
    df = gbo.DeviceBuffer.from_numpy(base)
    g.bmv_count(dx, df, gbo.OUT_F32, accumulate=True)
    assert np.array_equal(df.to_numpy(np.float32, n), base + want)
    do = gbo.DeviceBuffer(np.dtype(gbo.WORD_DTYPE[b]).itemsize * len(xw))
    for one in (n - 1, b * tiles - 1):  # found by the last item of the long row, or not at all
        ow = orc.pack_vector((np.arange(n) == one).astype(np.int32), b)
        g.bmv_masked(gbo.DeviceBuffer.from_numpy(ow.astype(gbo.WORD_DTYPE[b])), None, do)
        assert np.array_equal(do.to_numpy(gbo.WORD_DTYPE[b], len(xw)),
                              orc.bmv_masked(ref, ow, None).astype(gbo.WORD_DTYPE[b]))
    lab = rng.permutation(n).astype(np.int32)
    g.bmv_minselect(gbo.DeviceBuffer.from_numpy(lab), dy)
    assert np.array_equal(dy.to_numpy(np.int32, n), orc.bmv_minselect(ref, lab))
    g.bmv_minplus(gbo.DeviceBuffer.from_numpy(lab.astype(np.uint32)), dy)
    assert np.array_equal(dy.to_numpy(np.uint32, n), orc.bmv_minplus(ref, lab.astype(np.uint32)))
    xf = rng.integers(0, 8, n).astype(np.float32)
    dxf = gbo.DeviceBuffer.from_numpy(xf)
    row = np.repeat(np.arange(n), np.diff(csr.rowptr))
    sums = np.bincount(row, weights=xf[csr.colind], minlength=n)
    g.bmv_float(dxf, dy, 1.0, None, 0.0)
    assert np.array_equal(dy.to_numpy(np.float32, n), sums.astype(np.float32))


@pytest.mark.parametrize("b", [4, 8, 16])
def test_counts_of_rows_of_one_length(gbo, orc, gpu, b):
    """Every block row is cut, none is longer than the others: a warp counts one."""
    n = 200 * b + b // 2 + 1
    rng = np.random.default_rng(b)
    row = np.repeat(np.arange(n), 160)
    key = np.unique(row * np.int64(n) + rng.integers(0, n, len(row)))
    key = key[(key // n) // b != 7]  # one block row is empty
    rowptr = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(key // n, minlength=n), out=rowptr[1:])
    csr = gbo.Csr(rowptr, (key % n).astype(np.int32), n, n)
    g, ref = gbo.Graph.from_csr(csr, b), orc.pack(csr.rowptr, csr.colind, n, n, b)
    assert g.info().nsplit_rows == g.info().nblockrows - 1
    xw = orc.pack_vector((rng.random(n) < 0.5).astype(np.int32), b)
    dx = gbo.DeviceBuffer.from_numpy(xw.astype(gbo.WORD_DTYPE[b]))
    want = orc.bmv_count(ref, xw)
    dy = gbo.DeviceBuffer.from_numpy(np.full(n, -7, np.int32))
    g.bmv_count(dx, dy)
    assert np.array_equal(dy.to_numpy(np.int32, n), want)
    g.bmv_count(dx, dy, accumulate=True)
    assert np.array_equal(dy.to_numpy(np.int32, n), 2 * want)
    df = gbo.DeviceBuffer.from_numpy(np.full(n, 0.5, np.float32))
    g.bmv_count(dx, df, gbo.OUT_F32, accumulate=True)
    assert np.array_equal(df.to_numpy(np.float32, n), want + np.float32(0.5))
