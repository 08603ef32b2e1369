"""In-place shortest paths from a caller's own starting distances, at the sizes of the pull
rounds over the weight-sorted copy and of the persistent kernel, against the loop of
shortest_path! on the oracle's product.  Sums are whole numbers: comparisons are exact."""
import numpy as np
import pytest
import torch

import gpugraphs as G
from gpugraphs.multigraph import MultiGraph
from oracle import oracle as O
from test_graph_gpu import _reference_inplace
from test_search_queue_gpu import _graph

pytestmark = pytest.mark.gpu


def _starts(n, dtype, seed, lo, hi):
    """Two iterates with values in [lo, hi) at a third of the vertices each."""
    rng = np.random.default_rng(seed)
    top = np.inf if np.issubdtype(dtype, np.floating) else np.iinfo(dtype).max
    out = []
    for _ in range(2):
        d = rng.integers(lo, hi, n).astype(dtype)
        d[rng.random(n) < 0.67] = top
        out.append(d)
    return out


def _check(n, rp, cv, nz, source, dist0, next0):
    ref = _reference_inplace(n, rp, cv, nz, source, dist0, next0)
    A = G.SparseGPUMatrixCSR(n, n, rp, cv, nz)
    for _ in range(2):  # the second search finds the copies built
        d, x = torch.from_numpy(dist0).cuda(), torch.from_numpy(next0).cuda()
        G.shortest_path_(A, source, d, x)
        assert (d.cpu().numpy() == ref).all() and (x.cpu().numpy() == ref).all()


@pytest.mark.parametrize("dtype", [np.int32, np.bool_, np.float32])
@pytest.mark.parametrize("lo", [-200, 0])
@pytest.mark.parametrize("n", [12500, 70001])
def test_hub_graphs(n, lo, dtype):
    rng = np.random.default_rng(n)
    r, c = rng.integers(0, n, 9 * n), rng.integers(0, n, 9 * n)
    r, c = np.concatenate([r, np.full(700, 1)]), np.concatenate([c, rng.permutation(n)[:700]])
    keep = r != c
    rp, cv, nz = _graph(n, r[keep], c[keep], dtype, seed=2)
    if dtype != np.bool_:  # wide weights: a row's light entries come first in the sorted copy
        e = np.repeat(np.arange(n), np.diff(rp))
        h = (np.minimum(e, cv - 1).astype(np.int64) * 7919 + np.maximum(e, cv - 1) * 104729) % 255
        nz = (h + 1).astype(dtype)
    dd = np.int32 if dtype == np.bool_ else dtype
    dist0, next0 = _starts(n, dd, n + lo, lo, 200)
    _check(n, rp, cv, nz, 3, dist0, next0)


@pytest.mark.parametrize("dtype", [np.int32, np.int64, np.float32, np.float64])
@pytest.mark.parametrize("n", [2047, 2048, 3001, 70001])
def test_hub_free_graphs(n, dtype):
    """Single-CTA rounds below 2048 vertices, the persistent kernel from there."""
    v = np.arange(n)
    r, c = np.concatenate([v, v]), np.concatenate([(v + 1) % n, (v + 57) % n])
    rp, cv, nz = _graph(n, r, c, dtype, seed=4)
    dist0, next0 = _starts(n, dtype, n, -60, 60)
    _check(n, rp, cv, nz, n // 2, dist0, next0)


@pytest.mark.parametrize("dtype,scale", [(np.int32, 10**8), (np.int64, 10**17), (np.float32, 1e30)])
@pytest.mark.parametrize("n", [2048, 5000])
def test_heavy_weights(n, scale, dtype):
    """Mean weights whose multiple, the near-far band, is past the distance type."""
    rng = np.random.default_rng(n)
    v = np.arange(n)
    r, c = np.concatenate([v] * 6), np.concatenate([rng.permutation(n) for _ in range(6)])
    keep = r != c
    rp, cv, nz = _graph(n, r[keep], c[keep], dtype, seed=9)
    nz = (np.minimum(nz, 4) * dtype(scale)).astype(dtype)
    A = G.SparseGPUMatrixCSR(n, n, rp, cv, nz)
    ref, _ = O.sssp(n, rp, cv, nz, [1, n])
    for q, s in enumerate((1, n)):
        assert (G.shortest_path(A, s).cpu().numpy() == ref[:, q]).all()


@pytest.mark.parametrize("dtype", [np.int64, np.float64])
def test_starts_far_apart(dtype):
    """1400 paths of three vertices whose starts lie 2^52 apart: the gaps take more empty
    bands than eight a vertex (the first round, a product, reaches the middle vertices)."""
    n = 4200
    v = np.arange(0, n, 3)
    rp, cv, nz = _graph(n, np.concatenate([v, v + 1]), np.concatenate([v + 1, v + 2]), dtype)
    nz[:] = 1
    top = np.inf if dtype == np.float64 else np.iinfo(dtype).max
    dist0 = np.full(n, top, dtype)
    dist0[::3] = np.arange(n // 3).astype(dtype) * dtype(2**52)
    _check(n, rp, cv, nz, 1, dist0, dist0.copy())


def test_far_apart_in_many_graphs():
    """A dense graph of light edges beside a path of heavy ones: the path's steps are far
    wider than the common band."""
    n, m, p, w = 2000, 1 << 25, 6000, 2**40
    gen = torch.Generator(device="cuda").manual_seed(5)
    rowptr = (torch.arange(n + 1, device="cuda") * m // n + 1).to(torch.int32)
    cols = (torch.randint(0, n, (m,), generator=gen, device="cuda") + 1).to(torch.int32)
    dense = G.SparseGPUMatrixCSR(n, n, rowptr, cols, torch.ones(m, dtype=torch.int64, device="cuda"))
    v = np.arange(p - 1)
    rp, cv, nz = _graph(p, v, v + 1, np.int64)
    nz[:] = w
    d = MultiGraph([dense, G.SparseGPUMatrixCSR(p, p, rp, cv, nz)]).sssp([1, 1]).cpu().numpy()
    assert (d[n:] == np.arange(p) * w).all()
    assert d[0] == 0 and set(d[1:n]) == {1}
