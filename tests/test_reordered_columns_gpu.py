"""Products at the number of columns past which x is reordered by how often it is gathered."""
import numpy as np
import pytest
import torch

import gpugraphs as G

pytestmark = pytest.mark.gpu


def csr(m, n, dtype, seed):
    """Rows of 0 to 7 entries and three others; half the entries in 1000 columns."""
    rng = np.random.default_rng(seed)
    deg = rng.integers(0, 8, m)
    deg[[0, m // 2, m - 1]] = 300, 5000, 0
    rp = np.concatenate([[1], 1 + np.cumsum(deg)]).astype(np.int32)
    cv = rng.integers(1, n + 1, rp[-1] - 1).astype(np.int32)
    cv[::2] = cv[::2] % 1000 + 1
    nz = rng.integers(1, 100, len(cv))
    return rp, cv, (nz % 2 > 0) if dtype == np.bool_ else nz.astype(dtype)


@pytest.mark.parametrize("n", [1 << 20, (1 << 20) + 1])
@pytest.mark.parametrize("dtype", [np.int32, np.float32, np.float64, np.bool_])
@pytest.mark.parametrize("sell", [False, True])
def test_products_at_the_line_of_reordered_columns(n, dtype, sell):
    m = 70001
    rp, cv, nz = csr(m, n, dtype, 5)
    A = G.SparseGPUMatrixCSR(m, n, rp, cv, nz)
    if sell:
        A = G.SparseGPUMatrixSELL(A, 32, m)
    rng = np.random.default_rng(6)
    x = rng.integers(0, 1000, n)
    x = x % 3 == 0 if dtype == np.bool_ else x.astype(dtype)
    mask = rng.random(m) < 0.5
    live = np.diff(rp) > 0
    at = (rp[:-1] - 1)[live]
    if dtype == np.bool_:
        op, empty = dict(mul=G.GPUGraphs_band, add=G.GPUGraphs_bor), False
        folded = np.logical_or.reduceat(nz & x[cv - 1], at)
    else:
        op = dict(mul=G.GPUGraphs_safe_add, add=G.GPUGraphs_min)
        empty = np.iinfo(dtype).max if dtype == np.int32 else np.inf
        folded = np.minimum.reduceat(nz + x[cv - 1], at)
    want = np.full(m, empty, dtype)
    want[live] = folded
    for mk in (None, mask):
        y = torch.zeros(m, dtype=torch.from_numpy(want).dtype, device="cuda")
        kw = dict(op) if mk is None else dict(op, mask=torch.from_numpy(mk).cuda())
        G.gpu_spmv_(y, A, torch.from_numpy(x).cuda(), **kw)
        assert np.array_equal(y.cpu().numpy(), want if mk is None else np.where(mk, want, np.zeros_like(want)))
    if sell:  # a row range passes over the slices outside it
        y = torch.zeros(m, dtype=torch.from_numpy(want).dtype, device="cuda")
        G.gpu_spmv_(y, A, torch.from_numpy(x).cuda(), range=(30000, 36001), **op)
        ref = np.zeros_like(want)
        ref[29999:36001] = want[29999:36001]
        assert np.array_equal(y.cpu().numpy(), ref)
