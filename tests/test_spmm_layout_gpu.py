"""Column-major SpMM operands: the transposed routes against the oracle, over column
counts at the edges of tiles and vector loads, leading dimensions past the rows, masks,
row ranges, accumulators, element types, and hub rows cut into pieces."""
import numpy as np
import pytest
import torch

import gpugraphs as G
from oracle import oracle as O
from test_spmv_typed_gpu import matrix, values

pytestmark = pytest.mark.gpu


def colmajor(a, ld, shift=0):
    """A torch view of `a` inside a larger column-major block."""
    r, c = a.shape
    base = torch.zeros((c + 2, ld + shift), dtype=torch.from_numpy(a).dtype, device="cuda")
    view = base.T[shift:shift + r, 1:1 + c]
    view.copy_(torch.from_numpy(a).cuda())
    assert view.stride(0) == 1
    return view, base


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 31, 32, 33, 70])
@pytest.mark.parametrize("m,n", [(40, 37), (3001, 2999)])
@pytest.mark.parametrize("sel", ["all", "mask", "range"])
def test_float32_plus_times(k, m, n, sel):
    rp, cv, rng = matrix(m, n, True, 3) if m > 100 else matrix(200, n, True, 3)
    m = len(rp) - 1
    nz = values(rng, np.float32, len(cv))
    B = rng.random((n, k), dtype=np.float32)
    C0 = rng.random((m, k), dtype=np.float32)
    mask = rng.random(m) < 0.5 if sel == "mask" else None
    rg = (17, m - 5) if sel == "range" else None
    ref = np.asfortranarray(C0.copy())
    assert O.csr_spmm(m, rp, cv, nz, ref, np.asfortranarray(B), mask=mask, range_=rg) == O.OK
    A = G.SparseGPUMatrixCSR(m, n, rp, cv, nz)
    Bv, _ = colmajor(B, n + 3)
    for shift in (0, 1):
        Cv, base = colmajor(C0, m + 5, shift)
        before = base.clone()
        G.gpu_spmm_(Cv, A, Bv, mask=None if mask is None else torch.from_numpy(mask).cuda(), range=rg)
        got = Cv.cpu().numpy()
        short = np.diff(rp) <= 256
        assert (got[short] == ref[short]).all()
        np.testing.assert_allclose(got, ref, rtol=1e-5, atol=1e-5)
        Cv.copy_(torch.from_numpy(C0).cuda())
        assert torch.equal(base, before)  # nothing outside the view was written


@pytest.mark.parametrize("dtype,mul,add,acc", [
    (np.int32, "safe_add", "min", "min"), (np.bool_, "land", "lor", "second"),
    (np.float64, "mul", "add", "second"), (np.int64, "mul", "max", "max"),
    (np.float32, "mul", "add", "max"), (np.int32, "secondj", "add", "second")])
@pytest.mark.parametrize("k", [2, 33])
def test_other_semirings(dtype, mul, add, acc, k):
    m, n = 2500, 2601
    rp, cv, rng = matrix(m, n, True, 4)
    nz = values(rng, dtype, len(cv))
    tc = np.int64 if mul == "secondj" else dtype
    B = np.stack([values(rng, dtype, n) for _ in range(k)], 1)
    C0 = np.stack([values(rng, tc, m) for _ in range(k)], 1)
    code = {x: getattr(O, x.upper()) for x in (mul, add, acc)}
    op = {x: getattr(G, "GPUGraphs_" + x) for x in (mul, add, acc)}
    for mask in (None, rng.random(m) < 0.5):
        ref = np.asfortranarray(C0.copy())
        assert O.csr_spmm(m, rp, cv, nz, ref, np.asfortranarray(B), mul=code[mul], add=code[add],
                          accum=code[acc], mask=mask) == O.OK
        A = G.SparseGPUMatrixCSR(m, n, rp, cv, nz)
        for M in (A, G.SparseGPUMatrixSELL(A, 32, 64)):
            Cv, _ = colmajor(C0, m + 1)
            Bv, _ = colmajor(B, n)
            G.gpu_spmm_(Cv, M, Bv, mul=op[mul], add=op[add], accum=op[acc],
                        mask=None if mask is None else torch.from_numpy(mask).cuda())
            got = Cv.cpu().numpy()
            if np.issubdtype(dtype, np.floating):
                np.testing.assert_allclose(got, ref, rtol=1e-5, atol=1e-5)
            else:
                assert (got == ref).all()


@pytest.mark.parametrize("k", [2, 3, 5, 31, 33, 70])
@pytest.mark.parametrize("sel", ["all", "mask", "range"])
def test_row_major_of_odd_widths(k, sel):
    """Row-major rows that are no whole 16-byte groups, at an odd address and stride."""
    m, n = 3001, 2999
    rp, cv, rng = matrix(m, n, True, 5)
    nz = values(rng, np.float32, len(cv))
    B, C0 = rng.random((n, k), dtype=np.float32), rng.random((m, k), dtype=np.float32)
    mask = rng.random(m) < 0.5 if sel == "mask" else None
    rg = (17, m - 5) if sel == "range" else None
    ref = C0.copy()
    assert O.csr_spmm(m, rp, cv, nz, ref, B, layout=1, mask=mask, range_=rg) == O.OK
    A = G.SparseGPUMatrixCSR(m, n, rp, cv, nz)
    for shift, ld in ((0, k), (1, k + 2)):
        base = torch.zeros(m * ld + 3, dtype=torch.float32, device="cuda")
        Cv = base[shift:shift + m * ld].view(m, ld)[:, :k]
        Cv.copy_(torch.from_numpy(C0).cuda())
        before = base.clone()
        Bv = torch.zeros(n * ld + 3, dtype=torch.float32, device="cuda")[shift:shift + n * ld].view(n, ld)[:, :k]
        Bv.copy_(torch.from_numpy(B).cuda())
        G.gpu_spmm_(Cv, A, Bv, mask=None if mask is None else torch.from_numpy(mask).cuda(), range=rg)
        got = Cv.cpu().numpy()
        short = np.diff(rp) <= 256
        assert (got[short] == ref[short]).all()
        np.testing.assert_allclose(got, ref, rtol=1e-5, atol=1e-5)
        Cv.copy_(torch.from_numpy(C0).cuda())
        assert torch.equal(base, before)
