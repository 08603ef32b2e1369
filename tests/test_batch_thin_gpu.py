"""Batched shortest paths of graphs with few entries a row, most of whose rows are passed over
in most rounds: rows of 1 to 8 entries, longer ones among them, and pieces of a hub."""
import numpy as np
import pytest
import torch

import gpugraphs as G

pytestmark = pytest.mark.gpu


def graph(n, kind, dtype):
    r = np.arange(n - 1)
    c = r + 1
    if kind == "ladder":  # a path with rungs: entries of a row change in different rounds
        far = np.arange(0, n - 50, 3)
        r, c = np.append(r, far), np.append(c, far + 50)
    elif kind == "hubs":
        hub = np.arange(2, n - 1)
        nine = np.arange(n // 2 + 2, n // 2 + 10)
        r = np.concatenate([r, np.zeros(len(hub), int), np.full(8, n // 2)])
        c = np.concatenate([c, hub, nine])
    rng = np.random.default_rng(n)
    w = rng.integers(0, 100, len(r))
    i, j, v = np.append(r, c), np.append(c, r), np.append(w, w)
    order = np.lexsort((j, i))
    rp = np.concatenate([[1], 1 + np.cumsum(np.bincount(i, minlength=n))]).astype(np.int32)
    return G.SparseGPUMatrixCSR(n, n, rp, (j[order] + 1).astype(np.int32), v[order].astype(dtype))


@pytest.mark.parametrize("dtype", [np.int32, np.float32])
@pytest.mark.parametrize("kind", ["path", "ladder", "hubs"])
@pytest.mark.parametrize("n", [65, 1000, 3001])
def test_columns_equal_single_searches(n, kind, dtype):
    A = graph(n, kind, dtype)
    src = np.arange(40) * 7 % n + 1
    D = G.shortest_path(A, src)
    for q, s in enumerate(src):
        assert torch.equal(D[:, q], G.shortest_path(A, int(s)))
