"""PageRank-type loops over the row lists (merge-path parts) where the parts
can go wrong: rows over many parts, runs of empty rows, path lengths that are
whole multiples of a part, several parts per warp, every tile width; also the
loop after the graph's other traversals, and on two streams in turn."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
PART = 224  # items of a part (rows and set bits)


def _ring(gbo, n):
    return gbo.csr_from_edges(np.arange(n), (np.arange(n) + 1) % n, n, False, True)


def _star(gbo, n):
    return gbo.csr_from_edges(np.full(n - 1, n // 2), np.delete(np.arange(n), n // 2), n, True, True)


def _sparse_tail(gbo, n):
    """Edges among the first 700 vertices only: tens of thousands of empty rows."""
    rng = np.random.default_rng(1)
    return gbo.csr_from_edges(rng.integers(0, 700, 9000), rng.integers(0, 700, 9000), n, True, True)


GRAPHS = {
    "ring_one_part": lambda g: _ring(g, PART // 2),
    "ring_whole_parts": lambda g: _ring(g, PART // 2 * 57),
    "ring_part_and_one": lambda g: _ring(g, PART // 2 * 3 + 1),
    "star_hub": lambda g: _star(g, 300_001),
    "empty_rows": lambda g: _sparse_tail(g, 90_001),
    "many_parts": lambda g: g.gen_rmat(17, 16, seed=3),  # several parts a warp on any GPU
    "single": lambda g: g.csr_from_edges([0], [0], 1, False, False),
}


def _sum_rows(csr, terms):
    rows = np.repeat(np.arange(csr.nrows), np.diff(csr.rowptr))
    return np.bincount(rows, weights=terms[csr.colind], minlength=csr.nrows)


def _check(got, want):
    # three fp32 roundings an iteration, damped by 0.85: 3 * 2^-24 / 0.15
    assert np.abs(got - want).sum() <= 1.2e-6 * np.abs(want).sum()


@pytest.mark.parametrize("name", list(GRAPHS))
@pytest.mark.parametrize("b", [4, 32, 64])
def test_pagerank_parts(gbo, gpu, name, b):
    if b != 32 and name == "many_parts":
        pytest.skip("parts do not depend on the tile width")
    csr = GRAPHS[name](gbo)
    n = csr.nrows
    g = gbo.Graph.from_csr(csr, b)
    alpha = float(np.float32(0.85))
    deg = np.bincount(csr.colind, minlength=n).astype(np.float64)
    inv = np.divide(1.0, deg, out=np.zeros(n), where=deg > 0)
    p = np.full(n, 1.0 / n)
    for it in range(1, 6):
        p = alpha * _sum_rows(csr, p * inv) + (1 - alpha) / n
        got, iters = g.pagerank(alpha, it)
        assert iters == it
        _check(got.astype(np.float64), p)
    again, _ = g.pagerank(alpha, 5)
    assert np.array_equal(again, got)


@pytest.mark.parametrize("name", ["star_hub", "empty_rows", "many_parts"])
def test_ppr_and_adjoint_parts(gbo, gpu, name):
    csr = GRAPHS[name](gbo)
    n = csr.nrows
    g = gbo.Graph.from_csr(csr, 32, gbo.FLAG_SYMMETRIC)
    rng = np.random.default_rng(4)
    alpha = float(np.float32(0.85))
    v = rng.random(n).astype(np.float32)
    v /= v.sum()
    w = rng.standard_normal(n).astype(np.float32)
    deg = np.bincount(csr.colind, minlength=n).astype(np.float64)
    inv = np.divide(1.0, deg, out=np.zeros(n), where=deg > 0)
    p, u = (1 - alpha) * v.astype(np.float64), w.astype(np.float64)
    for _ in range(4):
        p = alpha * _sum_rows(csr, p * inv) + (1 - alpha) * v
        u = w + alpha * inv * _sum_rows(csr, u)
    g.bfs(0)  # the traversal's state and the loop's live in one handle
    _check(g.ppr_forward(v, alpha, -1.0, 4)[0].astype(np.float64), p)
    _check(g.ppr_backward(w, alpha, -1.0, 4)[0].astype(np.float64), (1 - alpha) * u)
    # a tolerance that stops at once, and one stream after another
    s = gbo.Stream()
    assert g.ppr_forward(v, alpha, 10.0, 50, stream=s.ptr)[1] == 1
    _check(g.ppr_forward(v, alpha, -1.0, 4)[0].astype(np.float64), p)


def test_injected_iteration_cap(gbo, gpu):
    g = gbo.Graph.from_csr(gbo.gen_rmat(10, 8, seed=1), 32)
    gbo.debug_inject(gbo.INJECT_REPLAY_CAP, 1)
    try:
        with pytest.raises(gbo.GboError) as e:
            g.pagerank(0.85, 100)
        assert e.value.status == gbo.GBO_ERR_TIMEOUT
    finally:
        gbo.debug_inject(gbo.INJECT_REPLAY_CAP, 0)
    assert g.pagerank(0.85, 100)[1] == 100


def test_loop_in_several_launches(gbo, gpu):
    """A loop holds the SMs for a bounded stretch: a large graph's iterations
    take several launches, with the same result and stopping point."""
    csr = gbo.gen_rmat(19, 16, seed=5)  # about 70,000 parts
    n = csr.nrows
    g = gbo.Graph.from_csr(csr, 32, gbo.FLAG_SYMMETRIC)
    alpha = float(np.float32(0.85))
    deg = np.bincount(csr.colind, minlength=n).astype(np.float64)
    inv = np.divide(1.0, deg, out=np.zeros(n), where=deg > 0)
    p = np.full(n, 1.0 / n)
    for _ in range(11):
        p = alpha * _sum_rows(csr, p * inv) + (1 - alpha) / n
    got, iters = g.pagerank(alpha, 11)
    stats = g.last_run()
    assert iters == 11 and stats["iterations"] == 11 and len(stats["step_ms"]) == 11
    assert 1 + 2 <= stats["kernel_launches"] <= 1 + 11  # the init kernel and the loop's
    _check(got.astype(np.float64), p)
    for tol in (1e-5, 1e-7):
        early, k = g.pagerank(alpha, 500, tol)
        assert 1 < k < 500
        assert np.array_equal(early, g.pagerank(alpha, k)[0])


def test_stream_with_a_part_of_the_sms(gbo, gpu):
    """A stream of a green context of 16 SMs refuses a grid of a block per SM:
    the loop runs on fewer blocks."""
    drv = pytest.importorskip("cuda.bindings.driver")

    def ok(r):
        if r[0] in (drv.CUresult.CUDA_ERROR_NOT_SUPPORTED, drv.CUresult.CUDA_ERROR_NOT_PERMITTED):
            pytest.skip("no green contexts here")
        assert r[0] == drv.CUresult.CUDA_SUCCESS, r[0]
        return r[1] if len(r) == 2 else r[1:]

    csr = gbo.gen_rmat(16, 16, seed=2)
    g = gbo.Graph.from_csr(csr, 32, gbo.FLAG_SYMMETRIC)
    want = g.pagerank(0.85, 7)[0]
    dev = ok(drv.cuDeviceGet(0))
    sms = ok(drv.cuDeviceGetDevResource(dev, drv.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    part = ok(drv.cuDevSmResourceSplitByCount(1, sms, 0, 16))[0]
    ctx = ok(drv.cuGreenCtxCreate(ok(drv.cuDevResourceGenerateDesc([part[0]], 1)), dev,
                                  drv.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    s = ok(drv.cuGreenCtxStreamCreate(ctx, drv.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    try:
        assert np.array_equal(g.pagerank(0.85, 7, stream=int(s))[0], want)
    finally:
        drv.cuStreamSynchronize(s)
        drv.cuStreamDestroy(s)
        drv.cuGreenCtxDestroy(ctx)
