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
