"""The device-built SELL-C-sigma arrays against the oracle's, bit for bit: slice heights
that do not divide the rows or cover them all, sort windows at the edges, rows far longer
than a fill tile, every element size."""
import numpy as np
import pytest

import gpugraphs as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.bool_, np.int32, np.float64])
@pytest.mark.parametrize("m,C,sigma", [(1, 32, 1), (33, 32, 33), (5000, 32, 1024), (5000, 7, 100),
                                       (5000, 1, 5000), (5000, 9000, 64), (70001, 32, 70001)])
def test_device_layout(dtype, m, C, sigma):
    n = 20000
    rng = np.random.default_rng(m + C)
    deg = rng.integers(0, 6, m)
    deg[rng.random(m) < 0.3] = 0
    deg[rng.integers(0, m, 3)] = [n // 2, 4097, 513][:3]
    rows = np.repeat(np.arange(m, dtype=np.int64), deg)
    key = np.unique(rows * n + rng.integers(0, n, len(rows)))
    rp = np.ones(m + 1, np.int32)
    rp[1:] += np.cumsum(np.bincount(key // n, minlength=m)).astype(np.int32)
    cv = (key % n + 1).astype(np.int32)
    nz = (rng.integers(0, 100, len(cv)) > 20) if dtype == np.bool_ else rng.integers(1, 99, len(cv)).astype(dtype)
    ref = O.sell_build(m, rp, cv, nz, slice_size=C, sigma=sigma)
    S = G.SparseGPUMatrixSELL(G.SparseGPUMatrixCSR(m, n, rp, cv, nz), C, sigma)
    assert S.n_stored == ref["n_stored"] and S.nslices == ref["nslices"]
    for name in ("slice_ptr", "colval", "nzval", "perm"):
        assert (getattr(S, name).cpu().numpy() == ref[name]).all(), name
