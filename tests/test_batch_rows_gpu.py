"""Batched shortest paths by weight-sorted rows: the light phase and the round that visits
every row after it, rows at the edges of the 8-entry steps and of the 256-entry pieces,
hubs of many pieces, even, equal, zero and infinite weights, and every value type.  Each
column equals the single-source distances, which other tests hold to Dijkstra's."""
import numpy as np
import pytest
import torch

import gpugraphs as G
from gpugraphs import generators as gen
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def graph(n, dtype, kind, seed):
    """Symmetric: hubs 0..19 of 7, 8, 9, 31, 32, 33, 255, 256, 257, 511, 513, 3000 ... edges."""
    rng = np.random.default_rng(seed)
    r, c = rng.integers(0, n, 9 * n), rng.integers(0, n, 9 * n)
    for h, d in enumerate([7, 8, 9, 31, 32, 33, 255, 256, 257, 511, 513, 3000, n // 2]):
        r = np.concatenate([r, np.full(d, n - 1 - h)])
        c = np.concatenate([c, rng.choice(n, d, replace=False)])
    lo, hi = np.minimum(r, c), np.maximum(r, c)
    key = np.unique((lo * n + hi)[lo != hi])
    w = {"even": rng.integers(1, 256, len(key)), "equal": np.full(len(key), 5),
         "zeros": rng.integers(0, 3, len(key)) * 9,
         "spread": np.floor(10.0 ** rng.uniform(0, 6, len(key)))}[kind].astype(np.float64)
    lo, hi = key // n, key % n
    rows, cols = np.concatenate([lo, hi]), np.concatenate([hi, lo])
    order = np.lexsort((cols, rows))
    rp = np.ones(n + 1, np.int32)
    rp[1:] += np.cumsum(np.bincount(rows, minlength=n)).astype(np.int32)
    return rp, (cols[order] + 1).astype(np.int32), np.concatenate([w, w])[order].astype(dtype)


@pytest.mark.parametrize("dtype", [np.bool_, np.int32, np.float32, np.int64, np.float64])
@pytest.mark.parametrize("kind", ["even", "equal", "zeros", "spread"])
@pytest.mark.parametrize("n,S", [(8000, 1), (8000, 33), (70001, 70)])
def test_columns_equal_single_sources(dtype, kind, n, S):
    if S == 1:  # a batch of one goes to the single-source engine: two sources, one column each
        S = 2
    rp, cv, nz = graph(n, dtype, kind, 5)
    A = G.SparseGPUMatrixCSR(n, n, rp, cv, nz)
    src = np.random.default_rng(6).integers(1, n + 1, S)
    src[0] = n  # a hub
    for M in (A, G.SparseGPUMatrixSELL(A, 32, 64)) if n < 10000 else (A,):
        D = G.shortest_path(M, src)
        for q in (0, S // 2, S - 1):
            assert torch.equal(D[:, q], G.shortest_path(A, int(src[q]))), q
    if dtype in (np.bool_, np.int32, np.float32):
        ref = O.sssp_dijkstra(n, rp, cv, nz, int(src[-1]), symmetric=True)
        assert (D[:, S - 1].cpu().numpy() == ref).all()


def test_many_groups_on_a_power_law_graph():
    A = gen.rmat(17, 16, seed=3, wkind=gen.W_INT_1_255)
    src = np.random.default_rng(1).integers(1, A.n + 1, 300)
    D = G.shortest_path(A, src)
    for q in list(range(0, 300, 29)) + [255, 256, 299]:
        assert torch.equal(D[:, q], G.shortest_path(A, int(src[q]))), q
