"""Searches at the sizes where the staged queue appends, the 128-edge push steps, the
hub pieces and the pull levels' bitmap-to-queue conversion can go wrong.  Levels and
distances are integers or exact fixpoints, so every comparison is exact."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

import gpugraphs as G
from oracle import oracle as O
from helpers import csr_from_scipy

pytestmark = pytest.mark.gpu


def _graph(n, r, c, dtype, seed=0):
    w = np.random.default_rng(seed).integers(1, 9, len(r)).astype(dtype)
    A = sp.coo_matrix((np.concatenate([w, w]), (np.concatenate([r, c]), np.concatenate([c, r]))),
                      shape=(n, n)).tocsr()
    return csr_from_scipy(A.astype(dtype))


def _check(n, rp, cv, nz, source):
    A = G.SparseGPUMatrixCSR(n, n, rp, cv, nz)
    pat = np.ones(len(cv), np.bool_)
    B = G.SparseGPUMatrixCSR(n, n, rp, cv, pat)
    lev, _ = O.bfs_levels_fast(n, rp, cv, pat, source, symmetric=True)
    dist = O.sssp_dijkstra(n, rp, cv, nz, source, symmetric=True)
    dist = dist[0] if isinstance(dist, tuple) else dist
    for _ in range(2):
        assert (G.bfs_distances(B, source).cpu().numpy() == lev).all()
        assert (G.shortest_path(A, source).cpu().numpy() == dist.reshape(-1)).all()


@pytest.mark.parametrize("n", [20000, 70001])
@pytest.mark.parametrize("deg", [31, 96, 97, 128, 129, 511, 512, 513, 1025, 9001])
def test_hub_with_leaves(n, deg):
    """source - hub - `deg` leaves - one more vertex each."""
    hub, leaf = 1, np.arange(2, 2 + deg)
    last = leaf + deg if 2 + 2 * deg <= n else leaf
    r = np.concatenate([[0], np.full(deg, hub), leaf])
    c = np.concatenate([[hub], leaf, last])
    keep = r != c
    _check(n, *_graph(n, r[keep], c[keep], np.int32, seed=deg), 1)


@pytest.mark.parametrize("tail", [1, 40])
@pytest.mark.parametrize("core", [3000, 66000, 70013])
def test_dense_core_then_paths(core, tail):
    """A random core (pull levels) with 33 paths hanging off it (push levels after)."""
    rng = np.random.default_rng(core + tail)
    r, c = rng.integers(0, core, 8 * core), rng.integers(0, core, 8 * core)
    p = core + np.arange(33 * tail).reshape(33, tail)
    prev = np.concatenate([rng.integers(0, core, (33, 1)), p[:, :-1]], axis=1)
    r, c = np.concatenate([r, prev.ravel()]), np.concatenate([c, p.ravel()])
    keep = r != c
    n = core + 33 * tail
    _check(n, *_graph(n, r[keep], c[keep], np.int32, seed=tail), 1 + int(r[keep][0]))
    _check(n, *_graph(n, r[keep], c[keep], np.float32, seed=tail), n)


@pytest.mark.parametrize("n,deg", [(65536, 3), (80001, 12), (1000003, 5)])
def test_hub_free_persistent_steps(n, deg):
    """Hub-free graphs (degrees of 1 to ~40): the persistent BFS / near-far kernels with
    vertices of more than 4 edges, and steps that append more than a block stages."""
    rng = np.random.default_rng(n)
    r, c = rng.integers(0, n, deg * n), rng.integers(0, n, deg * n)
    keep = r != c
    rp, cv, nz = _graph(n, r[keep], c[keep], np.float32, seed=deg)
    assert np.diff(rp).max() <= 64
    _check(n, rp, cv, nz, 1 + int(r[keep][0]))


@pytest.mark.parametrize("dtype", [np.bool_, np.int32, np.int64, np.float32, np.float64])
@pytest.mark.parametrize("sizes", [(2, 33, 700, 1500), (1, 1, 40000)])
def test_many_graphs_uneven_weights(dtype, sizes):
    """Several graphs at once: weights spread over nine decades, a vertex of 600 edges,
    isolated vertices, and result vectors that change between calls."""
    from gpugraphs.multigraph import MultiGraph
    gs, src, ref = [], [], []
    for i, n in enumerate(sizes):
        rng = np.random.default_rng(n + i)
        r, c = rng.integers(0, n, 3 * n), rng.integers(0, n, 3 * n)
        r, c = np.concatenate([r, np.zeros(min(n, 600), np.int64)]), np.concatenate([c, np.arange(min(n, 600))])
        r, c = r[r != c], c[r != c]
        lo, hi = np.minimum(r, c), np.maximum(r, c)
        key = np.unique(lo * n + hi) if len(lo) else np.zeros(0, np.int64)
        w = np.floor(10.0 ** rng.uniform(0, 6 if dtype == np.int32 else 9, len(key)))
        lo, hi = key // n, key % n
        A = sp.coo_matrix((np.concatenate([w, w]), (np.concatenate([lo, hi]), np.concatenate([hi, lo]))),
                          shape=(n, n)).tocsr()
        rp, cv, nz = csr_from_scipy(A.astype(dtype))
        gs.append(G.SparseGPUMatrixCSR(n, n, rp, cv, nz))
        src.append(n // 2 + 1)
        ref.append(G.shortest_path(gs[-1], n // 2 + 1).cpu().numpy())
        if dtype in (np.bool_, np.int32, np.float32):
            d = O.sssp_dijkstra(n, rp, cv, nz, n // 2 + 1, symmetric=True)
            assert (ref[-1] == d).all()
    mg = MultiGraph(gs)
    keep = []
    for _ in range(3):
        keep.append(mg.sssp(src))
        lev = mg.bfs(src) if dtype != np.float64 else None
        keep.append(lev)
    for out in keep[::2]:
        for got, want in zip(mg.split(out), ref):
            assert (got.cpu().numpy() == want).all()


@pytest.mark.parametrize("dtype", [torch.int32, torch.float32])
def test_many_graphs_in_bands(dtype):
    """More than 2^25 entries: near-far bands over all graphs, with weights of nine decades
    in one of them (empty bands, a band below the threshold's rounding)."""
    from gpugraphs import generators as gen
    from gpugraphs.multigraph import MultiGraph
    gs = []
    for i, n in enumerate((1100000, 3001, 50000)):
        A = gen.erdos_renyi(n, 16, seed=i + 3, symmetric=True, wkind=gen.W_INT_1_255)
        w = A.nzval.to(torch.float64)
        if i == 1:
            w = torch.floor(w ** (2.0 if dtype == torch.int32 else 3.7))
        gs.append(G.SparseGPUMatrixCSR(n, n, A.rowptr, A.colval, w.to(dtype)))
    assert sum(g.nnz() for g in gs) > 1 << 25
    src = [5, 3001, 7]
    mg = MultiGraph(gs)
    for _ in range(2):
        for got, A, s in zip(mg.split(mg.sssp(src)), gs, src):
            assert torch.equal(got, G.shortest_path(A, s))


@pytest.mark.parametrize("dtype", [np.bool_, np.int32, np.float32, np.float64, np.int64])
@pytest.mark.parametrize("kind", ["spread", "zeros", "equal", "infinite"])
def test_pull_rounds_stop_at_weights(dtype, kind):
    """Shortest paths through pull rounds whose rows are scanned by ascending weight:
    zero weights (-0.0 among them), equal ones, nine decades, +Inf, and hub rows of
    several chunks; distances equal Dijkstra's bit for bit, from several sources."""
    n = 70001
    rng = np.random.default_rng(11)
    r = rng.integers(0, n, 9 * n)
    c = np.where(rng.random(9 * n) < 0.3, rng.integers(0, 40, 9 * n), rng.integers(0, n, 9 * n))
    lo, hi = np.minimum(r, c), np.maximum(r, c)
    key = np.unique((lo * n + hi)[lo != hi])
    w = {"spread": np.floor(10.0 ** rng.uniform(0, 6, len(key))),
         "zeros": rng.integers(0, 3, len(key)) * 7.0,
         "equal": np.full(len(key), 3.0),
         "infinite": rng.integers(1, 50, len(key)).astype(float)}[kind]
    lo, hi = key // n, key % n
    rows, cols = np.concatenate([lo, hi]), np.concatenate([hi, lo])
    order = np.lexsort((cols, rows))
    vals = np.concatenate([w, w])[order]
    if kind == "zeros" and np.issubdtype(dtype, np.floating):
        vals = np.where(vals == 0, -0.0, vals)
    if kind == "infinite" and np.issubdtype(dtype, np.floating):
        edge = np.minimum(rows, cols)[order] * n + np.maximum(rows, cols)[order]
        vals = np.where(edge % 5 == 0, np.inf, vals)
    rp = np.ones(n + 1, np.int32)
    rp[1:] += np.cumsum(np.bincount(rows, minlength=n)).astype(np.int32)
    cv, nz = (cols[order] + 1).astype(np.int32), vals.astype(dtype)
    assert np.diff(rp).max() > 1000
    A = G.SparseGPUMatrixCSR(n, n, rp, cv, nz)
    for s in (1, 35000):
        got = G.shortest_path(A, s).cpu().numpy()
        if dtype in (np.bool_, np.int32, np.float32):
            assert (got == O.sssp_dijkstra(n, rp, cv, nz, s, symmetric=True)).all()
        else:  # whole numbers below 2^24: the 64-bit types' distances are the Float32 ones
            ref = O.sssp_dijkstra(n, rp, cv, nz.astype(np.float32), s, symmetric=True).astype(np.float64)
            exact = ref < 2 ** 24
            far = got.astype(np.float64) if dtype == np.float64 else np.where(got == np.iinfo(dtype).max, np.inf, got.astype(np.float64))
            assert (far[exact] == ref[exact]).all() and np.array_equal(np.isinf(far), np.isinf(ref))
