"""Packing of slabs with many entries (k_pack_wide): byte-exact against the
oracle at the sizes where its windows, unrolled walk and row runs end, and
the error paths inside such slabs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
WIDTHS = [4, 8, 16, 32, 64]


def _csr(rows, ncols):
    ptr = np.zeros(len(rows) + 1, np.int32)
    ptr[1:] = np.cumsum([len(r) for r in rows])
    return ptr, np.concatenate([np.asarray(r, np.int32) for r in rows])


def _pack(gbo, ptr, col, nrows, ncols, b, layout, shift=0):
    """Raw pack on caller-owned buffers; the tile array `shift` bytes into its
    allocation."""
    lib = gbo.lib()
    drp, dci = gbo.DeviceBuffer.from_numpy(ptr), gbo.DeviceBuffer.from_numpy(col)
    brp = gbo.DeviceBuffer(4 * ((nrows + b - 1) // b + 1))
    nb = gbo.C.c_int(0)
    gbo.check(lib.gbo_b2sr_nnzb(drp.ptr, dci.ptr, nrows, ncols, len(col), b, brp.ptr, gbo.C.byref(nb), None), "nnzb")
    wb = np.dtype(gbo.WORD_DTYPE[b]).itemsize
    bci, val = gbo.DeviceBuffer(4 * nb.value), gbo.DeviceBuffer.zeros(wb * b * nb.value + shift + 16)
    val.fill_bytes(0xA5)
    gbo.check(lib.gbo_b2sr_pack(drp.ptr, dci.ptr, nrows, ncols, len(col), b, layout, brp.ptr, bci.ptr,
                                val.ptr + shift, None), "pack")
    raw = val.to_numpy(np.uint8)
    assert (raw[:shift] == 0xA5).all() and (raw[shift + wb * b * nb.value:] == 0xA5).all()
    words = raw[shift:shift + wb * b * nb.value].view(gbo.WORD_DTYPE[b])
    return brp.to_numpy(np.int32), bci.to_numpy(np.int32, nb.value), words


# rows of one slab: runs of one column up to a full tile row, rows without
# entries, duplicates, a last column in a partial tile
@pytest.mark.parametrize("b", WIDTHS)
@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("ncols", [130, 5000, 40001])
def test_wide_slabs_match_oracle(gbo, orc, gpu, b, layout, ncols):
    rng = np.random.default_rng(ncols + b)
    rows = []
    for i in range(3 * b + 1):
        k = [0, 1, 129, ncols // 3, ncols][int(rng.integers(0, 5))] if i % b else ncols
        r = np.sort(rng.choice(ncols, size=min(k, 4200), replace=False)) if k < ncols else np.arange(min(ncols, 9000))
        rows.append(np.concatenate([r, [ncols - 1, ncols - 1]]) if i % 3 == 0 else r)
    rows = [np.sort(r) for r in rows]
    ptr, col = _csr(rows, ncols)
    ref = orc.pack(ptr, col, len(rows), ncols, b, layout)
    for shift in ((0, 4) if b < 64 else (0, 8)) + ((1,) if b <= 8 else ()):
        brp, bci, words = _pack(gbo, ptr, col, len(rows), ncols, b, layout, shift)
        assert np.array_equal(brp, ref.rowptr)
        assert np.array_equal(bci, ref.colind)
        assert np.array_equal(words, ref.narrow())


@pytest.mark.parametrize("b", [4, 64])
def test_block_columns_past_one_window(gbo, orc, gpu, b):
    """More block columns than the bitmap holds (about 0.9 M): further windows."""
    ncols = 1_000_003 * b
    rng = np.random.default_rng(b)
    rows = [np.unique(rng.integers(0, ncols, 700)) for _ in range(b + 2)]
    rows[1] = np.concatenate([rows[1][rows[1] < ncols - 9], np.arange(ncols - 9, ncols)])
    ptr, col = _csr(rows, ncols)
    for layout in (0, 1):
        ref = orc.pack(ptr, col, len(rows), ncols, b, layout)
        brp, bci, words = _pack(gbo, ptr, col, len(rows), ncols, b, layout)
        assert np.array_equal(brp, ref.rowptr) and np.array_equal(bci, ref.colind)
        assert np.array_equal(words, ref.narrow())


@pytest.mark.parametrize("b", WIDTHS)
def test_errors_inside_a_wide_slab(gbo, gpu, b):
    ncols = 4000
    good = [np.arange(0, ncols, 2) for _ in range(b)]
    for edit, status in ((lambda r: np.concatenate([r[:700], r[699:700] - 1, r[700:]]), gbo.GBO_ERR_UNSORTED),
                         (lambda r: np.concatenate([r, [ncols]]), gbo.GBO_ERR_BOUNDS),
                         (lambda r: np.concatenate([[-1], r]), gbo.GBO_ERR_BOUNDS)):
        rows = list(good)
        rows[b // 2] = edit(rows[b // 2])
        ptr, col = _csr(rows, ncols)
        with pytest.raises(gbo.GboError) as e:
            _pack(gbo, ptr, col, b, ncols, b, 0)
        assert e.value.status == status
    ptr, col = _csr(good, ncols)
    ptr[b // 2] = ptr[b // 2 + 1] + 1  # a row that ends before it starts
    with pytest.raises(gbo.GboError) as e:
        _pack(gbo, ptr, col, b, ncols, b, 0)
    assert e.value.status == gbo.GBO_ERR_BOUNDS


@pytest.mark.parametrize("nbc", [1_000_003, 2_100_000])
@pytest.mark.parametrize("b", [4, 16, 32, 64])
def test_errors_past_one_window(gbo, gpu, b, nbc):
    """Bad entries that no window's search returns: columns below the first and
    past the last block column, and (three windows) a stretch of a row moved so
    that the end of one window and the start of the next lie apart."""
    ncols = nbc * b - 3
    n = min(400, 4000 // b)  # a slab of one unit
    row = np.arange(n, dtype=np.int64) * ncols // n
    good = [row + i for i in range(b)]
    a, m = n // 20, n - n // 10
    bads = [(np.concatenate([row[a:m], row[:a], row[m:]]), gbo.GBO_ERR_UNSORTED),
            (np.concatenate([[-1], row]), gbo.GBO_ERR_BOUNDS),
            (np.concatenate([[-9 * b], row]), gbo.GBO_ERR_BOUNDS),
            (np.concatenate([row, [ncols]]), gbo.GBO_ERR_BOUNDS),
            (np.concatenate([row, [ncols + 3 + b]]), gbo.GBO_ERR_BOUNDS)]
    for bad, status in bads:
        rows = list(good)
        rows[b // 2] = bad
        ptr, col = _csr(rows, ncols)
        with pytest.raises(gbo.GboError) as e:
            _pack(gbo, ptr, col, b, ncols, b, 0)
        assert e.value.status == status
    ptr, col = _csr(good, ncols)
    _pack(gbo, ptr, col, b, ncols, b, 0)


@pytest.mark.parametrize("b", WIDTHS)
@pytest.mark.parametrize("ncols", [1500, 60_001, 3_000_000])
def test_slabs_on_both_sides_of_the_rules(gbo, orc, gpu, b, ncols):
    """One graph of hub slabs, slabs about the rules' lines (steps against the
    bitmap's words, the share of all work, side-by-side rows as in a mesh) and
    short ones: every slab is packed alike whoever packs it."""
    rng = np.random.default_rng(b + ncols)
    words = (ncols + b - 1) // b // 32 + 1
    rows = []
    for slab in range(40):
        kind = slab % 5
        steps = [3, words, words // 8, 200, 60][kind] * int(rng.integers(1, 4))
        for i in range(b):
            if kind == 4:  # short rows side by side over a wide span
                at = np.concatenate([slab * b + i + np.arange(-1, 2) + d for d in (0, ncols // 2, ncols - 50 * b)])
                rows.append(np.unique(at[(at >= 0) & (at < ncols)]))
            else:
                k = min(max(2 * steps // b, 1), 20_000 // b + 40, ncols // 2)
                rows.append(np.unique(rng.integers(0, ncols, k)))
    ptr, col = _csr(rows, ncols)
    for layout in (0, 1):
        ref = orc.pack(ptr, col, len(rows), ncols, b, layout)
        brp, bci, out = _pack(gbo, ptr, col, len(rows), ncols, b, layout)
        assert np.array_equal(brp, ref.rowptr) and np.array_equal(bci, ref.colind)
        assert np.array_equal(out, ref.narrow())


@pytest.mark.parametrize("b", [4, 8])
def test_fill_time_is_linear_in_the_graph(gbo, gpu, b):
    """A uniform graph four times as large takes about four times as long (16
    times when every slab walked a bitmap of all block columns)."""
    torch = pytest.importorskip("torch")

    def fill_ms(n):
        gen = torch.Generator(device="cuda").manual_seed(n)
        col = torch.randint(0, n, (n, 24), generator=gen, device="cuda", dtype=torch.int32).sort(1).values.flatten()
        ptr = torch.arange(0, 24 * n + 1, 24, device="cuda", dtype=torch.int32)
        rp = torch.empty((n + b - 1) // b + 1, dtype=torch.int32, device="cuda")
        nb = gbo.C.c_int(0)
        lib, args = gbo.lib(), (ptr.data_ptr(), col.data_ptr(), n, n, 24 * n, b)
        torch.cuda.synchronize()
        gbo.check(lib.gbo_b2sr_nnzb(*args, rp.data_ptr(), gbo.C.byref(nb), None), "nnzb")
        ci = torch.empty(nb.value, dtype=torch.int32, device="cuda")
        val = torch.empty(nb.value * b, dtype=torch.uint8, device="cuda")
        best = float("inf")
        for _ in range(4):
            a, z = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            gbo.check(lib.gbo_b2sr_pack(*args, 0, rp.data_ptr(), ci.data_ptr(), val.data_ptr(), None), "pack")
            z.record()
            z.synchronize()
            best = min(best, a.elapsed_time(z))
        return best

    assert fill_ms(1 << 21) < 12 * fill_ms(1 << 19)
