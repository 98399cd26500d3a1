"""Connected components where the sampled forest can go wrong: rows long enough
to be cut into chunks outside the largest component, a largest component whose
root is not the lowest vertex, components that meet at one root (links lost
and found again), long paths, no edges at all; repeated, since the links race."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _shuffle(rng, src, dst, n):
    p = rng.permutation(n)
    return p[src], p[dst]


def _stars(rng, n):
    """Three stars of 9,000, 8,000 and 5,000 leaves and isolated vertices."""
    src, dst, at = [], [], 3
    for hub, k in ((0, 9000), (1, 8000), (2, 5000)):
        src.append(np.full(k, hub))
        dst.append(np.arange(at, at + k))
        at += k
    return _shuffle(rng, np.concatenate(src), np.concatenate(dst), n)


def _low_bridge(rng, n):
    """A dense component on the high vertices; the low ones hang off it by
    single edges, so that its root moves in the last passes."""
    hi = rng.integers(n // 2, n, 8 * n)
    lo = np.arange(0, n // 2, 7)
    return np.concatenate([hi[::2], lo]), np.concatenate([hi[1::2], rng.integers(n // 2, n, len(lo))])


def _path(rng, n):
    return _shuffle(rng, np.arange(n - 1), np.arange(1, n), n)


def _sparse(rng, n):
    return rng.integers(0, n, n), rng.integers(0, n, n)


def _many(rng, n):
    """Dense graphs of 50 vertices each: no large component to sample."""
    a = rng.integers(0, n, 6 * n)
    return _shuffle(rng, a, a // 50 * 50 + rng.integers(0, 50, 6 * n) % np.minimum(50, n - a // 50 * 50), n)


def _none(rng, n):
    return np.zeros(0, np.int64), np.zeros(0, np.int64)


@pytest.mark.parametrize("make", [_stars, _low_bridge, _path, _sparse, _many, _none])
@pytest.mark.parametrize("n", [33, 30_001])
def test_labels_match_oracle(gbo, orc, gpu, make, n):
    if make is _stars:
        n = 30_001
    rng = np.random.default_rng(n)
    src, dst = make(rng, n)
    csr = gbo.csr_from_edges(src, dst, n, True, True)
    want = orc.cc(csr.rowptr, csr.colind, n)
    for b in (4, 32):
        g = gbo.Graph.from_csr(csr, b)
        for _ in range(10):
            assert np.array_equal(g.cc()[0], want)


def test_labels_without_waiting(gbo, orc, gpu):
    """h_iters NULL: queued on the caller's stream, no host wait."""
    csr = gbo.gen_rmat(13, 4, seed=5)
    g = gbo.Graph.from_csr(csr, 32)
    want = orc.cc(csr.rowptr, csr.colind, csr.nrows)
    s = gbo.Stream()
    out = gbo.DeviceBuffer(4 * csr.nrows)
    for _ in range(3):
        gbo.check(gbo.lib().gbo_cc(g.h, out.ptr, None, s.ptr), "cc")
        assert np.array_equal(out.to_numpy(np.int32, csr.nrows, s.ptr), want)


@pytest.mark.parametrize("kind,passes", [(0, 2), (5, 3), ("sparse", 3)])
def test_passes_and_their_times(gbo, gpu, kind, passes):
    """h_iters and the run's statistics tell the passes that ran: a star about
    vertex 0 is one tree after the first edges; about vertex 5 it is not (its
    second neighbour is taken there, 2 to 4 are left), nor is a sparse random
    graph."""
    n = 100_003
    rng = np.random.default_rng(3)
    src, dst = rng.integers(0, n, (2, 3 * n // 2)) if kind == "sparse" else (np.full(n, kind), np.arange(n))
    g = gbo.Graph.from_csr(gbo.csr_from_edges(src, dst, n, True, True), 32)
    assert g.cc()[1] == passes
    run = g.last_run()
    assert run["iterations"] == passes and len(run["step_ms"]) == passes
    assert min(run["step_ms"]) > 0 and run["kernel_launches"] >= 11
