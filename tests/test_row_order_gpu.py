"""The row order of SELL layouts, made on the host for few rows and on the device for more."""
import numpy as np
import pytest

import gpugraphs as G

pytestmark = pytest.mark.gpu


def csr(m):
    """Rows of 0 to 7 entries, two long ones and an empty last one."""
    rng = np.random.default_rng(m)
    deg = rng.integers(0, 8, m)
    if m > 100:
        deg[[0, m // 2, m - 1]] = 300, 5000, 0
    rp = np.concatenate([[1], 1 + np.cumsum(deg)]).astype(np.int32)
    return rp, rng.integers(1, m + 1, rp[-1] - 1).astype(np.int32)


@pytest.mark.parametrize("m,sigma", [(8192, 1000), (8193, 1000), (8192, 1 << 40), (8193, 8193),
                                     (32768, 1), (32769, 1), (31, 64), (1, 1), (3, 2)])
@pytest.mark.parametrize("C", [1, 7, 32])
def test_row_order(m, sigma, C):
    rp, cv = csr(m)
    S = G.SparseGPUMatrixSELL(G.SparseGPUMatrixCSR(m, m, rp, cv, np.ones(len(cv), np.float32)), C, sigma)
    length = np.diff(rp.astype(np.int64))
    window = np.arange(m) // sigma
    order = np.lexsort((np.arange(m), -length, window)) if sigma > 1 else np.arange(m)
    assert np.array_equal(S.perm.cpu().numpy(), order + 1)
    C = min(C, m)
    width = [length[order[t:t + C]].max() for t in range(0, m, C)]
    assert np.array_equal(S.slice_ptr.cpu().numpy(), 1 + np.concatenate([[0], np.cumsum(width)]) * C)
