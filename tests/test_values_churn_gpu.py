"""CSR and CSC handles whose values change: the SELL-32 copy costs some eight of the products it
speeds up, so after values that did not last it waits for the ninth: row blocks until then (one
launch; the copy's hub chunks take a second one), and either layout sees the new values."""
import pytest
import torch

import gpugraphs as G
from gpugraphs import generators as gen
from gpugraphs.tracing import launch_trace

pytestmark = pytest.mark.gpu
MINPLUS = dict(mul=G.GPUGraphs_safe_add, add=G.GPUGraphs_min)


@pytest.mark.parametrize("kind", ["csr", "csc"])
def test_copy_follows_how_long_values_last(kind):
    A = gen.rmat(17, 16, seed=3, wkind=gen.W_INT_1_255)  # symmetric: its own CSC arrays
    if kind == "csc":
        rp, cv, nz = (t.cpu().numpy() for t in (A.rowptr, A.colval, A.nzval))
        A = G.SparseGPUMatrixCSC(A.m, A.n, rp, cv, nz)
    ref = G.SparseGPUMatrixSELL(gen.rmat(17, 16, seed=3, wkind=gen.W_INT_1_255), 32, 1)
    x = torch.randint(0, 5000, (A.n,), device="cuda", dtype=torch.int32)
    shift = 0

    def launches(products):
        for _ in range(products):
            y, want = torch.zeros_like(x), torch.zeros_like(x)
            with launch_trace() as t:
                G.gpu_spmv_(y, A, x, **MINPLUS)
        G.gpu_spmv_(want, ref, x, **MINPLUS)
        want[want < 2**30] += shift  # every edge of a row is shift longer
        assert torch.equal(y, want)
        return t.launches

    def change():
        nonlocal shift
        shift += 3
        A.nzval.add_(3)
        A.values_changed()
    assert launches(1) == 2
    for _ in range(2):
        change()
        assert launches(1) == 1
    change()
    A.values_changed()  # several writes before the next product
    assert launches(8) == 1
    assert launches(1) == 2  # the ninth product makes the copy
    change()
    assert launches(7) == 2
    change()
    assert launches(1) == 1
