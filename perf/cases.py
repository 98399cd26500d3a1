"""Performance cases of the library: what its users call, over the range of
sizes, tile widths and graph shapes they call it with.

A case is a dict of plain values.  `listed()` names the standing cases,
`draw()` makes further ones of the same ranges, `prepare()` builds what a
program holds before the call (graph handle, vectors and output buffers on
the device), `run()` makes one pass through the public C ABI, `work()` states
the bytes and operations the pass cannot do without, and `exact()` gives the
floating-point results in 64 bits from torch alone.

Graphs are generated on the device from the seed:
  rmat  R-MAT (0.57, 0.19, 0.19), `ef` edges per vertex before symmetrising
        and deduplication: power-law degrees, hubs at low vertex numbers (as
        the library's own generator) or, with `shuffled`, anywhere
  er    uniformly random edges, average degree `ef`
  mesh  8-neighbour grid with 2 % of its edges missing: bounded degree, long
        diameter, dense tiles
`n` need not be a multiple of the tile width or a power of two.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "graph-bit-ops_b200"))
import gbo  # noqa: E402

ALPHA = float(np.float32(0.85))
WORD = {4: torch.uint8, 8: torch.uint8, 16: torch.int16, 32: torch.int32, 64: torch.int64}


def listed():
    return [
        # the smallest traversal: a 1,000-vertex random graph, where the call's
        # own latency (launches, level barriers, the depth read back) is all
        {"name": "bfs_er1000", "op": "bfs", "graph": "er", "n": 1000, "ef": 20, "b": 32},
        # the headline traversal: R-MAT scale 22, direction-optimising
        {"name": "bfs_rmat22", "op": "bfs", "graph": "rmat", "n": 1 << 22, "ef": 16, "b": 32},
        # 64 queries answered at once (one machine word pair per vertex)
        {"name": "msbfs64_rmat20", "op": "msbfs", "graph": "rmat", "n": 1 << 20, "ef": 16, "b": 32, "k": 64},
        # a full batch of a query server, not a multiple of the word size
        {"name": "msbfs1000_rmat17", "op": "msbfs", "graph": "rmat", "n": 1 << 17, "ef": 16, "b": 32, "k": 1000},
        # the standard ranking job: 20 iterations over a large graph
        {"name": "pagerank_rmat21", "op": "pagerank", "graph": "rmat", "n": 1 << 21, "ef": 16, "b": 32, "iters": 20},
        # forward and backward pass of personalized PageRank in a training step
        {"name": "ppr_rmat18", "op": "ppr", "graph": "rmat", "n": 1 << 18, "ef": 16, "b": 32, "iters": 30},
        # component labelling of a large graph whose vertex numbers say nothing
        # about degree, as edge lists from the field have them
        {"name": "cc_rmat20_shuffled", "op": "cc", "graph": "rmat", "n": 1 << 20, "ef": 16, "b": 32,
         "shuffled": True},
        # triangle count of a social-network-like graph
        {"name": "tc_rmat17", "op": "tc", "graph": "rmat", "n": 1 << 17, "ef": 16, "b": 32},
        # narrow tiles, the packing with the fewest bytes on sparse graphs
        {"name": "count_rmat20_b8", "op": "count", "graph": "rmat", "n": 1 << 20, "ef": 16, "b": 8},
        # fp32 product on a directed graph of an odd size (a user's own solver)
        {"name": "float_er1000003", "op": "float", "graph": "er", "n": 1000003, "ef": 24, "b": 32, "directed": True},
        # one masked Boolean step on a mesh-like graph (a user's own traversal)
        {"name": "masked_mesh701_b16", "op": "masked", "graph": "mesh", "n": 701 * 701, "ef": 8, "b": 16},
        # packing a graph that has just arrived on the device
        {"name": "pack_rmat19", "op": "pack", "graph": "rmat", "n": 1 << 19, "ef": 16, "b": 32},
    ]


def draw(rng):
    """One more case: the operations of the listed ones, sizes over their whole
    ranges (logarithmic, rarely round), every graph shape and the tile widths
    an operation takes."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def shape(lo, hi, kinds=("rmat", "rmat", "rmat", "er", "mesh")):
        kind = rng.choice(kinds)
        n = size(lo, hi)
        c = {"graph": kind, "n": n, "ef": rng.choice((8, 16, 24)) if kind != "mesh" else 8}
        if kind == "mesh":
            c["n"] = max(2, int(math.isqrt(n))) ** 2
        if kind == "rmat" and n <= 1 << 20 and rng.random() < 0.4:
            c["shuffled"] = True
        return c

    op = rng.choice(("bfs", "bfs", "msbfs", "pagerank", "pagerank", "ppr", "cc", "cc", "tc", "count", "count",
                     "float", "minplus", "minselect", "masked", "pack", "pack"))
    if op == "bfs":
        c = shape(1000, 1 << 22)
        c["b"] = rng.choice((32, 32, 32, 8, 16, 64)) if c["n"] <= 1 << 19 else 32
    elif op == "msbfs":
        c = shape(1000, 1 << 20, ("rmat", "rmat", "er"))
        # n * k levels, at most the 2^27 of the listed cases
        c.update(b=32, k=min(size(2, 1024), (1 << 27) // c["n"]))
    elif op in ("pagerank", "ppr"):
        c = shape(1000, (1 << 21) if op == "pagerank" else (1 << 18))
        c.update(b=rng.choice((32, 32, 32, 8)) if c["n"] <= 1 << 18 else 32, iters=rng.choice((10, 20, 30)))
        if op == "pagerank":
            c["iters"] = min(c["iters"], 20)
    elif op == "cc":
        c = shape(1000, 1 << 21)
        c["b"] = rng.choice((32, 32, 32, 8)) if c["n"] <= 1 << 18 else 32
    elif op == "tc":
        c = shape(1000, 1 << 17)
        c["b"] = rng.choice((8, 16, 32, 32))
    elif op == "pack":
        c = shape(1000, 1 << 19)
        c["b"] = rng.choice((4, 8, 16, 32, 32, 64)) if c["n"] <= 1 << 17 else rng.choice((4, 8, 16, 32))
        c["layout"] = rng.choice((0, 0, 1))
    else:
        c = shape(1000, 1 << 20)
        c["b"] = rng.choice((4, 8, 16, 32, 32, 64)) if c["n"] <= 1 << 19 else rng.choice((4, 8, 16, 32))
        c["directed"] = rng.random() < 0.5
        if op == "count":
            c["accumulate"] = rng.random() < 0.3
    c["op"] = op
    return c


# ------------------------------------------------------------------- inputs
def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + salt * 7919) % (1 << 62))
    return g


def _edges(case, seed):
    """Directed edge list (int64 source, destination) of the case's graph."""
    n, gen = case["n"], _gen(seed, 1)
    if case["graph"] == "rmat":
        bits = max(1, (n - 1).bit_length())
        m = n * case["ef"]
        src = torch.zeros(m, dtype=torch.int32, device="cuda")
        dst = torch.zeros(m, dtype=torch.int32, device="cuda")
        for _ in range(bits):
            r = torch.rand(m, generator=gen, device="cuda")
            src.mul_(2).add_(r >= 0.76)
            dst.mul_(2).add_(((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
        keep = (src < n) & (dst < n)
        src, dst = src[keep].long(), dst[keep].long()
        if case.get("shuffled"):
            perm = torch.randperm(n, generator=gen, device="cuda")
            src, dst = perm[src], perm[dst]
    elif case["graph"] == "er":
        m = n * case["ef"] // (1 if case.get("directed") else 2)
        src = torch.randint(0, n, (m,), generator=gen, device="cuda")
        dst = torch.randint(0, n, (m,), generator=gen, device="cuda")
    else:
        side = int(math.isqrt(n))
        v = torch.arange(n, device="cuda")
        y, x = v // side, v % side
        parts = []
        for dy, dx in ((0, 1), (1, -1), (1, 0), (1, 1)):
            ok = (y + dy < side) & (x + dx < side) & (x + dx >= 0)
            parts.append(torch.stack((v[ok], v[ok] + dy * side + dx)))
        e = torch.cat(parts, 1)
        e = e[:, torch.rand(e.shape[1], generator=gen, device="cuda") >= 0.02]
        src, dst = e[0], e[1]
    return src, dst


def _csr(case, seed):
    """CSR (int32 device tensors) of the case's graph: no self-loops, no
    duplicates, rows sorted; symmetric unless the case is directed."""
    n = case["n"]
    src, dst = _edges(case, seed)
    keep = src != dst
    src, dst = src[keep], dst[keep]
    if not case.get("directed"):
        src, dst = torch.cat((src, dst)), torch.cat((dst, src))
    key = torch.unique(src * n + dst)
    del src, dst
    row = torch.div(key, n, rounding_mode="floor")
    col = (key - row * n).int()
    ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    return ptr.int(), col


def _vectors(case, seed):
    """The case's dense input vectors (device tensors)."""
    n, gen, op = case["n"], _gen(seed, 2), case["op"]
    if op == "float":
        return {"x": torch.rand(n, generator=gen, device="cuda"),
                "scale": torch.rand(n, generator=gen, device="cuda") + 0.5}
    if op == "minplus":  # distances of a partly explored graph
        d = torch.randint(0, 64, (n,), generator=gen, device="cuda", dtype=torch.int32)
        d[torch.rand(n, generator=gen, device="cuda") < 0.4] = 2147483647
        return {"x": d}
    if op == "minselect":  # vertex labels
        return {"x": torch.randperm(n, generator=gen, device="cuda").int()}
    if op == "count":
        return {"bits": (torch.rand(n, generator=gen, device="cuda") < 0.5).int(),
                "y": torch.randint(0, 9, (n,), generator=gen, device="cuda", dtype=torch.int32)}
    if op == "masked":  # a frontier of a tenth of the vertices, a third visited
        return {"bits": (torch.rand(n, generator=gen, device="cuda") < 0.1).int(),
                "mask": (torch.rand(n, generator=gen, device="cuda") < 0.33).int()}
    if op == "ppr":  # a sparse personalization and a dense loss gradient
        v = torch.zeros(n, device="cuda")
        pick = torch.randperm(n, generator=gen, device="cuda")[:max(1, n // 100)]
        v[pick] = torch.rand(pick.shape[0], generator=gen, device="cuda") + 0.1
        return {"v": v / v.sum(), "w": torch.randn(n, generator=gen, device="cuda")}
    return {}


def _pack_bits(bits, b):
    n = bits.shape[0]
    words = torch.zeros((n + b - 1) // b, dtype=WORD[b], device="cuda")
    gbo.check(gbo.lib().gbo_pack_vector_i32(bits.data_ptr(), n, b, words.data_ptr(), None), "pack_vector")
    return words


def _graph(ptr, col, n, b, flags):
    h = C.c_void_p()
    gbo.check(gbo.lib().gbo_graph_from_csr(ptr.data_ptr(), col.data_ptr(), n, n, col.shape[0], b,
                                           flags | gbo.FLAG_DEVICE_PTRS, None, C.byref(h)), "graph_from_csr")
    return gbo.Graph(h.value)


def prepare(case, seed):
    op, n, b = case["op"], case["n"], case["b"]
    ptr, col = _csr(case, seed)
    s = {"case": case, "n": n, "b": b}
    s.update(_vectors(case, seed))
    nw = (n + b - 1) // b
    if op == "pack":
        # the program's buffers hold the most tiles there can be (one an entry)
        most = 2 * n * case["ef"]
        s.update(ptr=ptr, col=col, rowptr=torch.empty(nw + 1, dtype=torch.int32, device="cuda"),
                 colind=torch.zeros(most, dtype=torch.int32, device="cuda"),
                 words=torch.zeros(most * b, dtype=WORD[b], device="cuda"))
        torch.cuda.synchronize()
        return s
    flags = gbo.FLAG_LOWER if op == "tc" else 0 if case.get("directed") else gbo.FLAG_SYMMETRIC
    torch.cuda.synchronize()
    s["g"] = _graph(ptr, col, n, b, flags)
    if op in ("bfs", "msbfs"):  # sources: vertices with neighbours
        alive = torch.nonzero(ptr[1:] > ptr[:-1])[:, 0]
        pick = torch.randint(0, alive.shape[0], (case.get("k", 1),), generator=_gen(seed, 3), device="cuda")
        s["srcs"] = np.ascontiguousarray(alive[pick].cpu().numpy().astype(np.int32))
        s["level"] = torch.empty(n * case.get("k", 1), dtype=torch.int32, device="cuda")
    elif op in ("pagerank", "float"):
        s["out"] = torch.empty(n, dtype=torch.float32, device="cuda")
    elif op == "ppr":
        s["out"], s["grad"] = torch.empty(n, device="cuda"), torch.empty(n, device="cuda")
    elif op in ("cc", "minplus", "minselect"):
        s["out"] = torch.empty(n, dtype=torch.int32, device="cuda")
    elif op in ("count", "masked"):
        s["x"] = _pack_bits(s.pop("bits"), b)
        if op == "masked":
            s["mask"] = _pack_bits(s["mask"], b)
            s["out"] = torch.empty(nw, dtype=WORD[b], device="cuda")
        else:
            s["out"] = s.pop("y")
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    case, n, b, lib = s["case"], s["n"], s["b"], gbo.lib()
    op = case["op"]
    h = s["g"].h if "g" in s else None
    it = C.c_int(0)
    if op == "bfs":
        gbo.check(lib.gbo_bfs(h, int(s["srcs"][0]), s["level"].data_ptr(), C.byref(it), None), "bfs")
        return {"level": s["level"], "depth": it.value}
    if op == "msbfs":
        k = case["k"]
        gbo.check(lib.gbo_msbfs(h, s["srcs"].ctypes.data, k, s["level"].data_ptr(), C.byref(it), None), "msbfs")
        return {"level": s["level"].view(n, k), "depth": it.value}
    if op == "pagerank":
        gbo.check(lib.gbo_pagerank(h, ALPHA, case["iters"], -1.0, s["out"].data_ptr(), C.byref(it), None), "pagerank")
        return s["out"]
    if op == "ppr":
        gbo.check(lib.gbo_ppr_forward(h, s["v"].data_ptr(), ALPHA, -1.0, case["iters"], s["out"].data_ptr(),
                                      C.byref(it), None), "ppr_forward")
        gbo.check(lib.gbo_ppr_backward(h, s["w"].data_ptr(), ALPHA, -1.0, case["iters"], s["grad"].data_ptr(),
                                       C.byref(it), None), "ppr_backward")
        return {"p": s["out"], "grad": s["grad"]}
    if op == "cc":
        gbo.check(lib.gbo_cc(h, s["out"].data_ptr(), C.byref(it), None), "cc")
        return s["out"]
    if op == "tc":
        c = C.c_uint64(0)
        gbo.check(lib.gbo_tc(h, C.byref(c), None), "tc")
        return int(c.value)
    if op == "count":
        if case.get("accumulate"):  # onto counts the program already has, which it keeps
            y = s["out"].clone()
            gbo.check(lib.gbo_bmv_count(h, s["x"].data_ptr(), y.data_ptr(), gbo.OUT_I32, 1, None), "bmv_count")
            return y
        gbo.check(lib.gbo_bmv_count(h, s["x"].data_ptr(), s["out"].data_ptr(), gbo.OUT_I32, 0, None), "bmv_count")
        return s["out"]
    if op == "masked":
        gbo.check(lib.gbo_bmv_masked(h, s["x"].data_ptr(), s["mask"].data_ptr(), s["out"].data_ptr(), None),
                  "bmv_masked")
        return s["out"]
    if op == "float":
        gbo.check(lib.gbo_bmv_float(h, s["x"].data_ptr(), s["out"].data_ptr(), ALPHA, s["scale"].data_ptr(), 0.25,
                                    None), "bmv_float")
        return s["out"]
    if op == "minplus":
        gbo.check(lib.gbo_bmv_minplus(h, s["x"].data_ptr(), s["out"].data_ptr(), None), "bmv_minplus")
        return s["out"]
    if op == "minselect":
        gbo.check(lib.gbo_bmv_minselect(h, s["x"].data_ptr(), s["out"].data_ptr(), None), "bmv_minselect")
        return s["out"]
    # packing: the tile counts of the block rows, then the tiles
    nb = C.c_int(0)
    m = s["col"].shape[0]
    gbo.check(lib.gbo_b2sr_nnzb(s["ptr"].data_ptr(), s["col"].data_ptr(), n, n, m, b, s["rowptr"].data_ptr(),
                                C.byref(nb), None), "b2sr_nnzb")
    gbo.check(lib.gbo_b2sr_pack(s["ptr"].data_ptr(), s["col"].data_ptr(), n, n, m, b, case.get("layout", 0),
                                s["rowptr"].data_ptr(), s["colind"].data_ptr(), s["words"].data_ptr(), None),
              "b2sr_pack")
    return {"rowptr": s["rowptr"], "colind": s["colind"], "words": s["words"], "tiles": nb.value}


# ---------------------------------------------------- the pass's floor
def _entries(case):
    """Stored entries, about: the draws less the repeated ones."""
    n, ef = case["n"], case["ef"]
    if case["graph"] == "mesh":
        return int(7.8 * n)
    if case["graph"] == "er":
        return n * ef
    kept = 0.85 if n < 1 << 16 else 0.93
    return int(n * ef * kept * (1 if case.get("directed") else 2))


def work(case):
    """Every stored entry read once per sweep at four bytes (the smallest form
    a general sparse pattern has), vectors and results once."""
    n, nnz, op = case["n"], _entries(case), case["op"]
    it = case.get("iters", 1)
    if op == "bfs":  # a direction-optimising traversal: a parent per vertex, the levels
        return {"bytes": 12 * n, "flops": 0}
    if op == "msbfs":
        return {"bytes": 4 * nnz + 4 * n * case["k"], "flops": 0}
    if op == "pagerank":
        return {"bytes": it * (4 * nnz + 12 * n), "flops": it * 2 * nnz}
    if op == "ppr":
        return {"bytes": 2 * it * (4 * nnz + 12 * n), "flops": 4 * it * nnz}
    if op == "cc":
        return {"bytes": 4 * nnz + 8 * n, "flops": 0}
    if op == "tc":
        return {"bytes": 2 * nnz + 4 * n, "flops": 0}
    if op == "pack":  # the CSR in; at least one word and column per entry's tile out
        return {"bytes": 4 * nnz + 4 * n + 8 * nnz, "flops": 0}
    return {"bytes": 4 * nnz + 8 * n, "flops": 2 * nnz if op == "float" else 0}


# ------------------------------------------------- results in 64 bits
def _sum_rows(ptr, col, terms):
    """sum of terms[j] over the entries j of every row (fp64)."""
    n = ptr.shape[0] - 1
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), (ptr[1:] - ptr[:-1]).long())
    return torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, rows, terms[col.long()])


def exact(case, seed):
    op, n = case["op"], case["n"]
    if op not in ("pagerank", "ppr", "float"):
        return None  # whole numbers, compared as such
    ptr, col = _csr(case, seed)
    v = {k: t.double() for k, t in _vectors(case, seed).items()}
    if op == "float":
        return ALPHA * _sum_rows(ptr, col, v["x"] * v["scale"]) + 0.25
    deg = torch.bincount(col.long(), minlength=n).double()  # the graphs are symmetric
    inv = torch.where(deg > 0, 1.0 / deg.clamp(min=1), torch.zeros_like(deg))
    if op == "pagerank":
        p = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
        for _ in range(case["iters"]):
            p = ALPHA * _sum_rows(ptr, col, p * inv) + (1.0 - ALPHA) / n
        return p
    p = (1.0 - ALPHA) * v["v"]
    u = v["w"]
    for _ in range(case["iters"]):
        p = ALPHA * _sum_rows(ptr, col, p * inv) + (1.0 - ALPHA) * v["v"]
        u = v["w"] + ALPHA * inv * _sum_rows(ptr, col, u)
    return {"p": p, "grad": (1.0 - ALPHA) * u}
