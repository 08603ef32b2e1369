"""Products of the fixed semirings (matrix, operand and result of one type) on every
route: the SELL-32 copy of a large CSR (skewed and flat columns), row blocks (small
matrices, row ranges), SELL handles of several heights; masks, accumulators, rows at the
edges of the 8 / 32 / 128-entry groups, several chunks, and the stop at the absorbing
value with infinities and NaN.

Whole numbers, Bool and minima are compared bit for bit; sums of rows of at most 32 (CSR)
or 128 (SELL) entries too, longer ones within a bound of the products' absolute sum:
length x eps covers any order of the additions."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

import gpugraphs as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu

LENGTHS = [0, 0, 1, 1, 2, 3, 7, 8, 9, 31, 32, 33, 40, 127, 128, 129, 255, 256, 257, 1023, 1024,
           1025, 1152, 1153, 2500, 9000]


def matrix(m, n, skew, seed):
    """Rows of every length of LENGTHS (twice) among rows of 0..12 entries; columns drawn
    flat, or half of them among the first hundredth."""
    rng = np.random.default_rng(seed)
    deg = rng.integers(0, 13, m)
    at = rng.choice(m, 2 * len(LENGTHS), replace=False)
    deg[at] = np.minimum(LENGTHS * 2, n // 2)
    rows, cols = [np.repeat(np.arange(m), deg)], []
    flat = rng.integers(0, n, deg.sum())
    if skew:
        few = rng.integers(0, max(1, n // 100), len(flat))
        flat = np.where(rng.random(len(flat)) < 0.6, few, flat)
    key = np.unique(rows[0].astype(np.int64) * n + flat)
    r, c = key // n, key % n
    rowptr = np.ones(m + 1, np.int32)
    rowptr[1:] += np.cumsum(np.bincount(r, minlength=m)).astype(np.int32)
    return rowptr, (c + 1).astype(np.int32), rng


OPS = {"plustimes": (G.GPUGraphs_mul, G.GPUGraphs_add, O.MUL, O.ADD),
       "minplus": (G.GPUGraphs_safe_add, G.GPUGraphs_min, O.SAFE_ADD, O.MIN),
       "minadd": (G.GPUGraphs_add, G.GPUGraphs_min, O.ADD, O.MIN),
       "orand": (G.GPUGraphs_land, G.GPUGraphs_lor, O.LAND, O.LOR)}
CASES = [(np.bool_, "orand")] + [(t, s) for t in (np.int32, np.int64, np.float32, np.float64)
                                 for s in ("plustimes", "minplus", "minadd")]


def values(rng, dtype, n):
    if dtype == np.bool_:
        return rng.random(n) < 0.5
    return rng.integers(-40, 200, n).astype(dtype) if np.issubdtype(dtype, np.integer) else \
        (rng.random(n) * 3 - 1).astype(dtype)


def operand(rng, dtype, sr, n):
    x = values(rng, dtype, n)
    if sr != "orand":
        top = np.inf if np.issubdtype(dtype, np.floating) else np.iinfo(dtype).max
        if sr == "minplus":
            x[rng.random(n) < 0.3] = top
    return x


def check(M, m, n, rp, cv, nz, x, sr, dtype, mask, accum, y0, exact_len, rng_=None):
    mul, add, omul, oadd = OPS[sr]
    acc, oacc = {"second": (G.GPUGraphs_second, O.SECOND), "min": (G.GPUGraphs_min, O.MIN),
                 "max": (G.GPUGraphs_max, O.MAX)}[accum]
    ref = y0.copy()
    assert O.csr_spmv(m, n, rp, cv, nz, ref, x, omul, oadd, oacc, mask=mask, range_=rng_) == O.OK
    y = torch.from_numpy(y0.copy()).cuda()
    G.gpu_spmv_(y, M, torch.from_numpy(x).cuda(), mul=mul, add=add, accum=acc,
                mask=None if mask is None else torch.from_numpy(mask).cuda(), range=rng_)
    got = y.cpu().numpy()
    if sr == "plustimes" and np.issubdtype(dtype, np.floating):
        deg = np.diff(rp)
        A = sp.csr_matrix((np.abs(nz).astype(np.float64), cv - 1, rp - 1), shape=(m, n))
        bound = np.maximum(deg, 1) * np.finfo(dtype).eps * (A @ np.abs(x).astype(np.float64))
        short = deg <= exact_len
        if mask is not None:  # rows left out keep their value
            short = short | (mask == 0)
        same = (got == ref) | ((got != got) & (ref != ref))
        assert same[short].all()
        fin = ~short & np.isfinite(ref)
        assert (np.abs(got[fin] - ref[fin]) <= bound[fin]).all()
        assert same[~short & ~np.isfinite(ref)].all()
    else:
        assert ((got == ref) | ((got != got) & (ref != ref))).all()


@pytest.mark.parametrize("dtype,sr", CASES)
@pytest.mark.parametrize("m,n,skew", [(65536, 66000, True), (70001, 70001, False), (3001, 90000, True)])
def test_csr_routes(dtype, sr, m, n, skew):
    rp, cv, rng = matrix(m, n, skew, 7)
    nz = values(rng, dtype, len(cv))
    A = G.SparseGPUMatrixCSR(m, n, rp, cv, nz)
    for mask, accum in ((None, "second"), (rng.random(m) < 0.5, "second"), (None, "min"),
                        ((rng.random(m) < 0.02).astype(np.int32), "max")):
        y0 = values(rng, dtype, m)
        check(A, m, n, rp, cv, nz, operand(rng, dtype, sr, n), sr, dtype, mask, accum, y0, 32)
    check(A, m, n, rp, cv, nz, operand(rng, dtype, sr, n), sr, dtype, None, "second",
          values(rng, dtype, m), 32, rng_=(100, m // 2))


@pytest.mark.parametrize("dtype,sr", CASES)
@pytest.mark.parametrize("m,C,sigma", [(9001, 32, 1), (9001, 32, 1024), (9001, 8, 64),
                                       (65700, 32, 1), (65700, 16, 64), (65700, 32, 65700)])
def test_sell_routes(dtype, sr, m, C, sigma):
    """Own slices (small matrices, whole-matrix windows) and the sorted copy of padded ones."""
    n = 70000
    rp, cv, rng = matrix(m, n, True, 8)
    nz = values(rng, dtype, len(cv))
    S = G.SparseGPUMatrixSELL(G.SparseGPUMatrixCSR(m, n, rp, cv, nz), C, sigma)
    if m > 65536:
        assert S.n_stored > 1.25 * S.nnz()
    for mask, accum, rg in ((None, "second", None), (rng.random(m) < 0.5, "min", None),
                            (None, "max", (33, 4000))):
        check(S, m, n, rp, cv, nz, operand(rng, dtype, sr, n), sr, dtype, mask, accum,
              values(rng, dtype, m), 128, rng_=rg)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("sr", ["plustimes", "minplus", "minadd"])
@pytest.mark.parametrize("m", [66000, 5000])
def test_stop_at_the_absorbing_value(dtype, sr, m):
    """+Inf, -Inf and NaN in x: every row's result (NaN pattern included) is that of the
    sequential fold with its stop, masked as well."""
    n = 70000
    rp, cv, rng = matrix(m, n, True, 9)
    nz = np.abs(values(rng, dtype, len(cv))) + 1
    A = G.SparseGPUMatrixCSR(m, n, rp, cv, nz.astype(dtype))
    for frac in (0.001, 0.05):
        x = rng.random(n).astype(dtype)
        for v in (np.inf, -np.inf, np.nan):
            x[rng.random(n) < frac] = v
        for mask in (None, rng.random(m) < 0.5):
            check(A, m, n, rp, cv, nz.astype(dtype), x, sr, dtype, mask, "second",
                  np.zeros(m, dtype), 32)


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_whole_sums_stop_at_typemax(dtype):
    """A sum that reaches typemax exactly stops there (rows folded in storage order)."""
    m = n = 65600
    top = np.iinfo(dtype).max
    rp = (1 + 3 * np.arange(m + 1)).astype(np.int32)
    cv = (1 + (np.arange(3 * m) % n)).astype(np.int32)
    nz = np.tile(np.array([top - 5, 5, 9], dtype), m)
    x = np.ones(n, dtype)
    A = G.SparseGPUMatrixCSR(m, n, rp, cv, nz)
    check(A, m, n, rp, cv, nz, x, "plustimes", dtype, None, "second", np.zeros(m, dtype), 32)


@pytest.mark.parametrize("sigma", [1, 256])
def test_runtime_operators_on_the_sorted_copy(sigma):
    """A semiring without a fixed kernel (max of products) on a padded SELL handle, and new
    values after a first product."""
    m = n = 66001
    rp, cv, rng = matrix(m, n, True, 12)
    nz = rng.integers(1, 90, len(cv)).astype(np.int32)
    S = G.SparseGPUMatrixSELL(G.SparseGPUMatrixCSR(m, n, rp, cv, nz), 32, sigma)
    x = rng.integers(1, 90, n).astype(np.int32)
    ref = np.zeros(m, np.int32)
    assert O.csr_spmv(m, n, rp, cv, nz, ref, x, O.MUL, O.MAX, O.SECOND) == O.OK
    y = torch.zeros(m, dtype=torch.int32, device="cuda")
    G.gpu_spmv_(y, S, torch.from_numpy(x).cuda(), mul=G.GPUGraphs_mul, add=G.GPUGraphs_max)
    assert (y.cpu().numpy() == ref).all()
