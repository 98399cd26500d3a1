"""Triangle counts over lists of ranked neighbours: graphs of enough tiles to be
counted that way (each case checks that it is), at all tile widths -- lists of
several units and of several pieces, ranks past the bitmap, hubs, diagonal
entries, rows short enough for a lane each -- and a matrix with entries above
its diagonal, which is not counted that way.  Exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILES = 1 << 16  # from here on lists are built


def _edges(kind, n, rng):
    if kind == "mesh":  # at most 3 lower neighbours a row
        side = int(n ** 0.5)
        v = np.arange(side * side).reshape(side, side)
        pairs = [(v[:, 1:], v[:, :-1]), (v[1:], v[:-1]), (v[1:, 1:], v[:-1, :-1])]
        return np.concatenate([a.ravel() for a, _ in pairs]), np.concatenate([b.ravel() for _, b in pairs])
    src, dst = rng.integers(0, n, 8 * n), rng.integers(0, n, 8 * n)
    if kind == "sparse":
        return src[:n], dst[:n]
    # a clique of 300 (lists of up to 299), a hub over everything, triangles
    # among vertices of the lowest degrees, whose ranks are the highest
    clique = rng.permutation(n)[:300]
    a, b = np.triu_indices(300, 1)
    low = np.arange(n - 3000, n)
    keep = (src < n - 3000) & (dst < n - 3000)
    src = [src[keep], clique[a], np.full(n // 8, 17), low, low]
    dst = [dst[keep], clique[b], np.arange(n // 8), low // 3 * 3, (low + 1) // 3 * 3]
    return np.concatenate(src), np.concatenate(dst)


def _lower(gbo, kind, n, diagonal):
    rng = np.random.default_rng(n)
    src, dst = _edges(kind, n, rng)
    hi, lo = np.maximum(src, dst), np.minimum(src, dst)
    keep = hi > lo
    hi, lo = hi[keep], lo[keep]
    if diagonal:
        d = rng.permutation(n)[: n // 3]
        hi, lo = np.concatenate([hi, d]), np.concatenate([lo, d])
    key = np.unique(hi.astype(np.int64) * n + lo)
    rowptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(key // n, minlength=n), out=rowptr[1:])
    return rowptr.astype(np.int32), (key % n).astype(np.int32)


@pytest.mark.parametrize("diagonal", [False, True])
@pytest.mark.parametrize("kind,n,b", [("dense", 36_001, 4), ("dense", 36_001, 8), ("dense", 36_002, 16),
                                      ("dense", 36_001, 32), ("dense", 40_001, 64), ("sparse", 90_001, 8),
                                      ("mesh", 600_625, 32), ("mesh", 40_000, 4)])
def test_lists(gbo, orc, gpu, kind, n, b, diagonal):
    rowptr, colind = _lower(gbo, kind, n, diagonal)
    want = orc.tc_b2sr(orc.pack(rowptr, colind, n, n, b))
    g = gbo.Graph.from_csr(gbo.Csr(rowptr, colind, n, n), b)
    before = g.info()
    assert before.nblocks >= TILES or kind == "mesh" and b == 4
    for _ in range(2):
        assert g.tc() == want
    if before.nblocks >= TILES:
        assert g.info().device_bytes >= before.device_bytes + 4 * len(colind)


@pytest.mark.parametrize("b", [4, 32])
def test_entry_above_the_diagonal(gbo, orc, gpu, b):
    n = 40_001
    rowptr, colind = _lower(gbo, "dense", n, True)
    row = np.repeat(np.arange(n), np.diff(rowptr))
    key = np.unique(np.concatenate([row * n + colind, [5 * n + 39_000, 6 * n + 39_000]]))
    rowptr = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(key // n, minlength=n), out=rowptr[1:])
    colind = (key % n).astype(np.int32)
    g = gbo.Graph.from_csr(gbo.Csr(rowptr, colind, n, n), b)
    assert g.info().nblocks >= TILES
    assert g.tc() == orc.tc_b2sr(orc.pack(rowptr, colind, n, n, b))


@pytest.mark.parametrize("b", [8, 32])
def test_wrapped_graph_with_wrong_degrees(gbo, orc, gpu, b):
    """The out-degrees of a wrapped graph order the lists and no more: any
    numbers give the same count."""
    n = 36_001
    rowptr, colind = _lower(gbo, "dense", n, False)
    want = orc.tc_b2sr(orc.pack(rowptr, colind, n, n, b))
    rp, ci, words = gbo.Graph.from_csr(gbo.Csr(rowptr, colind, n, n), b).b2sr()
    rng = np.random.default_rng(b)
    deg = rng.choice(np.array([-2**31, -70_000, -1, 0, 1, 1023, 1024, 2**31 - 1]), n).astype(np.int32)
    bufs = [gbo.DeviceBuffer.from_numpy(a) for a in (rp, ci, words, deg)]
    g = gbo.Graph.wrap_b2sr(n, n, b, 0, len(ci), *bufs)
    assert g.info().nblocks >= TILES
    for _ in range(2):
        assert g.tc() == want


@pytest.mark.parametrize("kind,n,b,first", [("mesh", 700_569, 8, False), ("sparse", 90_001, 8, False),
                                            ("dense", 40_001, 64, True), ("sparse", 600_001, 8, True)])
def test_first_count_builds_where_it_pays(gbo, orc, gpu, kind, n, b, first):
    """A graph's first count goes over the tiles where building the lists would
    cost more; its second one builds them."""
    rowptr, colind = _lower(gbo, kind, n, False)
    want = orc.tc_b2sr(orc.pack(rowptr, colind, n, n, b))
    g = gbo.Graph.from_csr(gbo.Csr(rowptr, colind, n, n), b)
    before = g.info()
    assert before.nblocks >= TILES
    assert g.tc() == want
    lists = 4 * len(colind) + 8 * n
    assert (g.info().device_bytes >= before.device_bytes + lists) == first
    assert g.tc() == want
    assert g.info().device_bytes >= before.device_bytes + lists


@pytest.mark.parametrize("b", [4, 8, 16, 32, 64])
@pytest.mark.parametrize("where", ["diagonal_tile", "above_it"])
def test_one_entry_above_builds_nothing(gbo, orc, gpu, b, where):
    n = 40_001
    rowptr, colind = _lower(gbo, "dense", n, True)
    row = np.repeat(np.arange(n), np.diff(rowptr))
    at = b * (n // b // 2)
    extra = at * n + (at + b - 1 if where == "diagonal_tile" else at + b)
    key = np.unique(np.concatenate([row * np.int64(n) + colind, [extra]]))
    rowptr = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(key // n, minlength=n), out=rowptr[1:])
    colind = (key % n).astype(np.int32)
    want = orc.tc_b2sr(orc.pack(rowptr, colind, n, n, b))
    g = gbo.Graph.from_csr(gbo.Csr(rowptr, colind, n, n), b)
    before = g.info()
    for _ in range(3):
        assert g.tc() == want
    assert g.info().device_bytes == before.device_bytes + 4 * before.nblocks  # the tiles' block rows
