"""Triangle counts recorded by stream capture, before and after a direct count
of the graph, below and above the line of the neighbour lists: replays and
direct calls agree with the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lower(gbo, n, b):
    rng = np.random.default_rng(n + b)
    src, dst = rng.integers(0, n, 9 * n), rng.integers(0, n // 3, 9 * n)
    hi, lo = np.maximum(src, dst), np.minimum(src, dst)
    key = np.unique(hi[hi > lo].astype(np.int64) * n + lo[hi > lo])
    rowptr = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(key // n, minlength=n), out=rowptr[1:])
    return rowptr, (key % n).astype(np.int32)


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
@pytest.mark.parametrize("n,b,flags", [(900, 8, 0), (1200, 32, "mma"), (30_001, 8, 0), (30_001, 32, 0)])
def test_first_count_captured(gbo, orc, gpu, n, b, flags, mode):
    torch = pytest.importorskip("torch")
    rowptr, colind = _lower(gbo, n, b)
    want = orc.tc_b2sr(orc.pack(rowptr, colind, n, n, b))
    flags = gbo.FLAG_TC_MMA if flags == "mma" else 0
    other = gbo.Graph.from_csr(gbo.Csr(rowptr, colind, n, n), b, flags)
    g = gbo.Graph.from_csr(gbo.Csr(rowptr, colind, n, n), b, flags)
    count = torch.zeros(1, dtype=torch.int64, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()

    def record():
        rec = torch.cuda.CUDAGraph()
        with torch.cuda.graph(rec, stream=s, capture_error_mode=mode):
            gbo.check(gbo.lib().gbo_tc_device(g.h, count.data_ptr(), s.cuda_stream), "tc_device")
        return rec

    before = g.info().device_bytes
    first = record()
    assert g.info().device_bytes == before  # nothing recorded belongs to the handle
    assert other.tc() == want  # a direct count meanwhile
    assert g.tc() == want  # and one of the same graph before any replay
    for rec in (first, record()):
        for _ in range(2):
            count.fill_(-1)
            rec.replay()
            torch.cuda.synchronize()
            assert int(count.item()) == want
    assert g.tc() == want
