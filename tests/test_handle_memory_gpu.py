"""Device memory of a matrix goes with the matrix and the tensors over its arrays."""
import gc

import pytest
import torch

import gpugraphs as G
from gpugraphs import generators as gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["csr", "csc", "sell"])
def test_dropped_matrices_free_their_memory(kind):
    A = gen.rmat(18, 16, seed=1)  # about 60 MB
    rp, cv, nz = (t.cpu().numpy() for t in (A.rowptr, A.colval, A.nzval))
    make = {"csr": lambda: G.SparseGPUMatrixCSR(A.m, A.n, rp, cv, nz),
            "csc": lambda: G.SparseGPUMatrixCSC(A.m, A.n, rp, cv, nz),
            "sell": lambda: G.SparseGPUMatrixSELL(A, 32, 1024)}[kind]

    def used():
        gc.collect()
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[1] - torch.cuda.mem_get_info()[0]
    make()
    before = used()
    for _ in range(4):
        make()
    assert used() - before < 32 << 20  # less than one of them


def test_tensors_outlive_their_matrix():
    A = gen.grid(20, 20)
    colval, want = A.colval, A.colval.cpu()
    del A
    gc.collect()
    gen.grid(21, 21)
    assert torch.equal(colval.cpu(), want)
