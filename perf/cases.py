"""Performance cases: what a user of the package has it do, through its public calls.

Every graph and vector is made on the GPU from the seed alone: R-MAT (a=0.57, b=0.19,
c=0.19, d=0.05, edge factor 16, symmetrised, no self-loops, duplicates merged),
Erdos-Renyi (uniform edges, duplicates merged) and 4-neighbour grids, with values
uniform [0, 1), Int32 weights 1..255 or Float32 weights [1, 10)."""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.abspath("gpugraphs.jl_gb300"))
import gpugraphs as G  # noqa: E402
from gpugraphs.multigraph import MultiGraph  # noqa: E402

DEV = "cuda"
DTYPES = {"bool": torch.bool, "int32": torch.int32, "float32": torch.float32,
          "float64": torch.float64}


def listed():
    return [
        # a small sparse product: launch count and latency decide
        spmv("spmv_er_16k", graph="er", n=16384, degree=16, dtype="float32"),
        # the product of a large power-law graph (PageRank-like iterations, random walks)
        spmv("spmv_rmat22", graph="rmat", n=1 << 22, degree=16, dtype="float32"),
        # one Bellman-Ford round written with the semiring product, as user algorithms are
        spmv("spmv_minplus_rmat21", graph="rmat", n=1 << 21, degree=16, dtype="int32",
             semiring="minplus"),
        # one masked or-and step of a user-written search over Bool adjacency
        spmv("spmv_orand_mask_rmat20", graph="rmat", n=1 << 20, degree=16, dtype="bool",
             semiring="orand", mask=True),
        # double-precision iteration on the SELL-C-sigma storage
        spmv("spmv_sell_f64_rmat20", graph="rmat", n=1 << 20, degree=16, dtype="float64",
             slice_size=32, sigma=1024),
        # feature propagation: sparse times 32 dense columns, row-major
        spmm("spmm_row32_rmat22", n=1 << 22, k=32, layout="row"),
        # the same on Julia's column-major arrays
        spmm("spmm_col32_rmat20", n=1 << 20, k=32, layout="col"),
        # hop levels of one source in a large power-law graph
        search("bfs_rmat24", "bfs", graph="rmat", n=1 << 24, degree=16, dtype="bool"),
        # shortest paths of one source in a power-law graph
        search("sssp_rmat22", "sssp", graph="rmat", n=1 << 22, degree=16, dtype="int32"),
        # shortest paths on a road-like (high-diameter) graph
        search("sssp_grid2048", "sssp", graph="grid", n=2048 * 2048, width=2048,
               dtype="float32"),
        # all-sources-of-a-batch shortest paths: distances from 256 vertices at once
        batch("batch_sssp256_rmat20", "sssp", n=1 << 20, sources=256),
        # many independent uneven graphs, one search in each
        multi("multi_sssp_128", "sssp", graphs=128, n_max=200000),
    ]


def spmv(name=None, **kw):
    return _case(name, dict(op="spmv", semiring="plustimes", mask=False, slice_size=0, sigma=0), kw)


def spmm(name=None, **kw):
    return _case(name, dict(op="spmm", graph="rmat", degree=16, dtype="float32"), kw)


def search(name, kind, **kw):
    return _case(name, dict(op=kind), kw)


def batch(name, kind, **kw):
    return _case(name, dict(op="batch_" + kind, graph="rmat", degree=16,
                            dtype="int32" if kind == "sssp" else "bool"), kw)


def multi(name, kind, **kw):
    dtype = {"spmv": "float32", "bfs": "bool", "sssp": "int32"}[kind]
    return _case(name, dict(op="multi_" + kind, dtype=dtype), kw)


def _case(name, base, kw):
    c = dict(base, **kw)
    if name is not None:
        c["name"] = name
    return c


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above: every family, sizes log-uniform (odd ones and
    powers of two), the data types, semirings, masks and layouts that go with it."""
    family = rng.choice(["spmv", "spmv", "spmm", "search", "search", "batch", "multi"])
    if family == "spmv":
        graph = rng.choice(["rmat", "rmat", "er", "grid"])
        dtype, semiring = rng.choice([("float32", "plustimes"), ("float32", "plustimes"),
                                      ("float64", "plustimes"), ("int32", "minplus"),
                                      ("float32", "minplus"), ("bool", "orand")])
        kw = _graph(rng, graph, 1000, 1 << 22)
        C, sigma = rng.choice([(0, 0), (0, 0), (0, 0), (8, 64), (16, 1024), (32, 1024)])
        return spmv(dtype=dtype, semiring=semiring, mask=rng.random() < 0.3,
                    slice_size=C, sigma=sigma, **kw)
    if family == "spmm":
        return spmm(n=_size(rng, 1000, 1 << 20), k=rng.choice([1, 4, 8, 16, 31, 32, 64]),
                    layout=rng.choice(["row", "col"]))
    if family == "search":
        kind = rng.choice(["bfs", "sssp"])
        graph = rng.choice(["rmat", "rmat", "er", "grid"])
        dtype = "bool" if kind == "bfs" else rng.choice(["int32", "float32"])
        return search(None, kind, dtype=dtype, **_graph(rng, graph, 1000, 1 << 22))
    if family == "batch":
        return batch(None, rng.choice(["bfs", "sssp"]), n=_size(rng, 1 << 12, 1 << 20),
                     sources=_log(rng, 8, 256))
    return multi(None, rng.choice(["spmv", "bfs", "sssp"]), graphs=_log(rng, 8, 128),
                 n_max=_log(rng, 4000, 200000))


def _size(rng, lo, hi):
    n = _log(rng, lo, hi)
    return 1 << round(math.log2(n)) if rng.random() < 0.4 else n


def _graph(rng, graph, lo, hi):
    n = _size(rng, lo, hi)
    if graph == "grid":
        w = max(2, int(math.sqrt(n) * rng.uniform(0.7, 1.4)))
        return dict(graph="grid", n=w * max(2, n // w), width=w)
    return dict(graph=graph, n=n, degree=16)


# ---------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _rmat_edges(n, count, gen):
    src = torch.zeros(count, dtype=torch.int64, device=DEV)
    dst = torch.zeros(count, dtype=torch.int64, device=DEV)
    for _ in range(max(1, (n - 1).bit_length())):
        r = torch.rand(count, generator=gen, device=DEV)
        src = src * 2 + (r >= 0.76)
        dst = dst * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    if n & (n - 1):
        keep = (src < n) & (dst < n)
        src, dst = src[keep], dst[keep]
    return src, dst


def _assemble(n, src, dst, symmetric):
    """Sorted, duplicate-free keys row * 2^32 + column."""
    if symmetric:
        key = torch.cat([(src << 32) | dst, (dst << 32) | src])[torch.cat([src != dst] * 2)]
    else:
        key = (src << 32) | dst
    key = torch.sort(key).values
    if key.numel() > 1:
        first = torch.ones_like(key, dtype=torch.bool)
        first[1:] = key[1:] != key[:-1]
        key = key[first]
    return key


def _values(key, dtype, seed, low, high):
    """Values by undirected edge and seed, so a symmetric pattern has a symmetric matrix."""
    r, c = key >> 32, key & 0xFFFFFFFF
    h = torch.minimum(r, c) * 0x9E3779B97F4A7C1 + torch.maximum(r, c) * 0x2545F4914F6CDD1D
    h = h + seed * 0x5851F42D4C957F2D % (1 << 62)
    for _ in range(2):
        h = (h ^ ((h >> 29) & 0x7FFFFFFFF)) * 0x3C79AC492BA7B653
    bits = (h >> 32) & 0xFFFFFF
    if dtype == torch.bool:
        return torch.ones(key.numel(), dtype=torch.bool, device=DEV)
    if dtype == torch.int32:
        return (bits % 255 + 1).to(torch.int32)
    u = bits.to(dtype) * (1.0 / (1 << 24))
    return u if (low, high) == (0, 1) else u * (high - low) + low


def _pattern(case, seed, symmetric):
    gen = _gen(seed)
    if case["graph"] == "grid":
        n, W = case["n"], case["width"]
        v = torch.arange(n, device=DEV)
        right, down = v[(v % W) < W - 1], v[v < n - W]
        return gen, _assemble(n, torch.cat([right, down]), torch.cat([right + 1, down + W]), True)
    n, ne = case["n"], case["n"] * case["degree"]
    if case["graph"] == "rmat":
        src, dst = _rmat_edges(n, ne, gen)
        return gen, _assemble(n, src, dst, True)
    src = torch.randint(0, n, (ne,), generator=gen, device=DEV)
    dst = torch.randint(0, n, (ne,), generator=gen, device=DEV)
    return gen, _assemble(n, src, dst, symmetric)


def _entries(case, seed):
    """(generator, key, values): the stored entries in row-major order."""
    path = case["op"] in ("sssp", "batch_sssp", "bfs", "batch_bfs")
    weights = (1, 10) if path or case.get("semiring") == "minplus" else (0, 1)
    gen, key = _pattern(case, seed, symmetric=path)
    return gen, key, _values(key, DTYPES[case["dtype"]], seed, *weights)


def _csr(n, key, vals):
    rowptr = torch.ones(n + 1, dtype=torch.int32, device=DEV)
    rowptr[1:] += torch.cumsum(torch.bincount(key >> 32, minlength=n), 0).to(torch.int32)
    return G.SparseGPUMatrixCSR(n, n, rowptr, ((key & 0xFFFFFFFF) + 1).to(torch.int32), vals)


def _sources(key, count, gen):
    """Distinct-row draws (0-based) among the vertices that have an edge."""
    rows = torch.unique_consecutive(key >> 32)
    return rows[torch.randint(0, rows.numel(), (count,), generator=gen, device=DEV)]


def _operand(case, gen):
    n, dtype = case["n"], DTYPES[case["dtype"]]
    if case["semiring"] == "orand":
        return torch.rand(n, generator=gen, device=DEV) < 0.1
    if case["semiring"] == "minplus":  # distances of a search under way: half not reached
        d = torch.randint(0, 4096, (n,), generator=gen, device=DEV).to(dtype)
        far = torch.rand(n, generator=gen, device=DEV) < 0.5
        return torch.where(far, torch.full_like(d, _typemax(dtype)), d)
    return torch.rand(n, generator=gen, device=DEV, dtype=dtype)


def _typemax(dtype):
    return math.inf if dtype.is_floating_point else torch.iinfo(dtype).max


def _mask(case, gen):
    return torch.rand(case["n"], generator=gen, device=DEV) < 0.5 if case["mask"] else None


def _multi_sizes(case):
    """(n, edges) of every graph: n log-uniform in [1000, n_max], mean degree 4..32."""
    out = []
    for g in range(case["graphs"]):
        n = int(1000 * (case["n_max"] / 1000) ** (((g * 37) % case["graphs"]) / max(1, case["graphs"] - 1)))
        out.append((n, int(n * (2 + 14 * ((g * 0.6180339887) % 1.0)))))
    return out


def _multi_entries(case, seed):
    gen = _gen(seed)
    dtype = DTYPES[case["dtype"]]
    graphs = []
    for g, (n, ne) in enumerate(_multi_sizes(case)):
        src = torch.randint(0, n, (ne,), generator=gen, device=DEV)
        dst = torch.randint(0, n, (ne,), generator=gen, device=DEV)
        key = _assemble(n, src, dst, True)
        graphs.append((n, key, _values(key, dtype, seed + g, 0, 1)))
    return gen, graphs


def prepare(case, seed):
    s = {"case": case}
    op, n = case["op"], case.get("n")
    if op.startswith("multi_"):
        gen, graphs = _multi_entries(case, seed)
        s["A"] = MultiGraph([_csr(n, key, vals) for n, key, vals in graphs])
        if op == "multi_spmv":
            s["x"] = torch.rand(s["A"].total_n, generator=gen, device=DEV)
        else:
            s["sources"] = [int(_sources(key, 1, gen)) + 1 for _, key, _ in graphs]
        return s
    gen, key, vals = _entries(case, seed)
    A = _csr(n, key, vals)
    if op == "spmv":
        if case["slice_size"]:
            A = G.SparseGPUMatrixSELL(A, case["slice_size"], case["sigma"])
        s["x"] = _operand(case, gen)
        s["mask"] = _mask(case, gen)
        s["y"] = s["x"].clone()
        if case["semiring"] == "plustimes":
            s["op"] = dict(mul=G.GPUGraphs_mul, add=G.GPUGraphs_add)
        elif case["semiring"] == "minplus":
            s["op"] = dict(mul=G.GPUGraphs_safe_add, add=G.GPUGraphs_min, accum=G.GPUGraphs_min)
        else:
            s["op"] = dict(mul=G.GPUGraphs_band, add=G.GPUGraphs_bor)
    elif op == "spmm":
        x = torch.rand(n, case["k"], generator=gen, device=DEV)
        s["x"], s["y"] = (x, torch.zeros_like(x)) if case["layout"] == "row" else (
            x.T.contiguous().T, torch.zeros(case["k"], n, device=DEV).T)
    elif op.startswith("batch_"):
        s["sources"] = (_sources(key, case["sources"], gen) + 1).cpu().numpy()
    else:
        s["source"] = int(_sources(key, 1, gen)) + 1
    s["A"] = A
    return s


def run(s):
    op, A = s["case"]["op"], s["A"]
    if op == "spmv":
        G.gpu_spmv_(s["y"], A, s["x"], mask=s["mask"], **s["op"])
        return s["y"]
    if op == "spmm":
        G.gpu_spmm_(s["y"], A, s["x"])
        return s["y"]
    if op == "bfs":
        return G.bfs_distances(A, s["source"])
    if op == "sssp":
        return G.shortest_path(A, s["source"])
    if op == "batch_bfs":
        return G.bfs_distances_batch(A, s["sources"])
    if op == "batch_sssp":
        return G.shortest_path(A, s["sources"])
    if op == "multi_spmv":
        return A.spmv(s["x"])
    return A.bfs(s["sources"]) if op == "multi_bfs" else A.sssp(s["sources"])


# ---------------------------------------------------------------------------------
# work of one pass
# ---------------------------------------------------------------------------------

def _counts(case):
    """(rows, stored entries) to a few percent."""
    if case["op"].startswith("multi_"):
        sizes = _multi_sizes(case)
        return sum(n for n, _ in sizes), 2 * sum(ne for _, ne in sizes)
    n = case["n"]
    if case["graph"] == "grid":
        return n, 4 * n
    path = case["op"] in ("sssp", "bfs")
    if case["graph"] == "er":
        return n, (32 if path else 16) * n
    if n & (n - 1):
        p = 1 << (n - 1).bit_length()
        return n, int(32 * n * (0.8 + 0.15 * n / p))
    return n, int(32 * n * min(0.98, 0.956 + 0.007 * (math.log2(n) - 22)))


def work(case):
    """Matrix once, operands once, results once; 2 operations an entry and column."""
    n, nnz = _counts(case)
    e = torch.tensor([], dtype=DTYPES[case["dtype"]]).element_size()
    kind = case["op"].split("_")[-1]
    cols = {"spmm": case.get("k"), "bfs": case.get("sources", 1), "sssp": case.get("sources", 1)}.get(kind, 1)
    if kind == "bfs":
        return {"bytes": 4 * (n + 1) + 4 * nnz + 4 * n * cols, "flops": nnz * cols}
    if kind == "sssp":
        return {"bytes": 4 * (n + 1) + 8 * nnz + 4 * n * cols, "flops": 2 * nnz * cols}
    moved = 4 * (n + 1) + (4 + e) * nnz + 2 * e * n * cols
    if case.get("mask"):
        moved = 4 * (n + 1) + (4 + e) * nnz // 2 + 2 * e * n + n
    return {"bytes": moved, "flops": 2 * nnz * cols}


# ---------------------------------------------------------------------------------
# the same results in 64 bits by plain torch
# ---------------------------------------------------------------------------------

def _rows_cols(key):
    return key >> 32, key & 0xFFFFFFFF


def _product(n, key, vals, x):
    """sum over the entries of each row of value * x[column], in 64 bits."""
    r, c = _rows_cols(key)
    y = torch.zeros((n,) + tuple(x.shape[1:]), dtype=torch.float64, device=DEV)
    for lo in range(0, key.numel(), 1 << 24):
        part = slice(lo, lo + (1 << 24))
        v = vals[part].double().reshape((-1,) + (1,) * (x.dim() - 1))
        y.index_add_(0, r[part], v * x[c[part]].double())
    return y


def _grid_paths(case, key, vals, source):
    """Bellman-Ford on the grid's arrays of right and down weights."""
    n, W = case["n"], case["width"]
    H = n // W
    r, c = _rows_cols(key)
    east = torch.full((n,), math.inf, dtype=torch.float64, device=DEV)
    south = east.clone()
    east[r[c == r + 1]] = vals[c == r + 1].double()
    down = c == r + W
    south[r[down]] = vals[down].double()
    east, south = east.view(H, W)[:, :-1].contiguous(), south.view(H, W)[:-1].contiguous()
    d = torch.full((H, W), math.inf, dtype=torch.float64, device=DEV)
    d.view(-1)[source] = 0
    for step in range(n):
        before = d.clone() if step % 64 == 0 else None
        e = d.clone()
        e[:, 1:] = torch.minimum(e[:, 1:], d[:, :-1] + east)
        e[:, :-1] = torch.minimum(e[:, :-1], d[:, 1:] + east)
        e[1:] = torch.minimum(e[1:], d[:-1] + south)
        e[:-1] = torch.minimum(e[:-1], d[1:] + south)
        d = e
        if before is not None and torch.equal(before, d):
            break
    return d.view(-1)


def _paths(n, key, vals, source):
    r, c = _rows_cols(key)
    v = vals.double()
    d = torch.full((n,), math.inf, dtype=torch.float64, device=DEV)
    d[source] = 0
    while True:
        e = d.scatter_reduce(0, r, v + d[c], "amin")
        if torch.equal(e, d):
            return d
        d = e


def exact(case, seed):
    """None where the outputs are whole numbers or truth values."""
    op = case["op"]
    if case["dtype"] not in ("float32", "float64"):
        return None
    if op == "multi_spmv":
        gen, graphs = _multi_entries(case, seed)
        x = torch.rand(sum(n for n, _, _ in graphs), generator=gen, device=DEV)
        parts = x.split([n for n, _, _ in graphs])
        return torch.cat([_product(n, key, vals, xg) for (n, key, vals), xg in zip(graphs, parts)])
    gen, key, vals = _entries(case, seed)
    n = case["n"]
    if op == "spmm":
        y = _product(n, key, vals, torch.rand(n, case["k"], generator=gen, device=DEV))
        return y if case["layout"] == "row" else y.T.contiguous().T
    if op == "sssp":
        source = int(_sources(key, 1, gen))
        return _grid_paths(case, key, vals, source) if case["graph"] == "grid" else _paths(n, key, vals, source)
    x = _operand(case, gen)
    mask = _mask(case, gen)
    if case["semiring"] == "plustimes":
        y = _product(n, key, vals, x)
    else:
        r, c = _rows_cols(key)
        y = x.double().scatter_reduce(0, r, vals.double() + x.double()[c], "amin")
    return y if mask is None else torch.where(mask, y, x.double())
