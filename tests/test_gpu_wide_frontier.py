"""Multi-source BFS with frontier rows of 4 to 32 words at the edges of every
width: rows of 0, 1, 31, 32, 33, 255 to 257, 512, 513 and 5,000 columns (the
line past which a row is cut into chunks, and chunks' own edges), directed so
that levels pull from them, a ragged last block row; every column against one
oracle BFS."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 31, 32, 33, 255, 256, 257, 511, 512, 513, 5000]


@pytest.fixture(scope="module")
def graphs(gbo):
    rng = np.random.default_rng(7)
    n = 6007
    src = [np.full(m, 3 + 29 * i) for i, m in enumerate(LENGTHS)]
    dst = [rng.permutation(n)[:m] for m in LENGTHS]
    chain = np.arange(n - 1)  # so that every row is met
    src, dst = np.concatenate(src + [chain[::3]]), np.concatenate(dst + [chain[::3] + 1])
    return [gbo.csr_from_edges(src.astype(np.int32), dst.astype(np.int32), n, s, True) for s in (False, True)]


@pytest.mark.parametrize("k", [65, 128, 129, 256, 257, 512, 513, 1024])
def test_levels(gbo, orc, gpu, graphs, k):
    rng = np.random.default_rng(k)
    for csr, flags in zip(graphs, (0, gbo.FLAG_SYMMETRIC)):
        n = csr.nrows
        srcs = rng.integers(0, n, k).astype(np.int32)
        srcs[:len(LENGTHS)] = 3 + 29 * np.arange(len(LENGTHS))
        srcs[-1] = n - 1
        g = gbo.Graph.from_csr(csr, 32, flags)
        for _ in range(2):
            lv, depth = g.msbfs(srcs)
        want = np.stack([orc.bfs_csr(csr.rowptr, csr.colind, n, int(s))[0] for s in srcs], 1)
        assert np.array_equal(lv, want)
        assert depth == int(want.max()) + 1


def test_directed_graph_builds_no_slices(gbo, gpu, graphs):
    csr = graphs[0]
    g = gbo.Graph.from_csr(csr, 32)
    before = g.info().device_bytes
    g.msbfs(np.arange(100, dtype=np.int32))
    slices = 8 * 8 * csr.nrows  # their heads alone
    assert g.info().device_bytes < before + slices


@pytest.mark.parametrize("k", [60, 100, 1000])
def test_symmetry_asserted_between_calls(gbo, orc, gpu, graphs, k):
    """A graph that pulled at first pushes once it is said to be symmetric, and
    pulls again afterwards."""
    csr = graphs[1]
    n = csr.nrows
    srcs = np.arange(5, 5 + k, dtype=np.int32)
    want = np.stack([orc.bfs_csr(csr.rowptr, csr.colind, n, int(s))[0] for s in srcs], 1)
    g = gbo.Graph.from_csr(csr, 32)
    for symmetric, threshold in ((0, -1), (1, -1), (1, 100_000), (0, -1), (1, 50)):
        g.set_bfs_direction(symmetric, threshold)
        assert np.array_equal(g.msbfs(srcs)[0], want)
