"""Masked column-major SpMM of large operands: the rows a mask keeps are counted on the device,
and the product runs where B lies or through row-major scratch, never both (an accumulator
would show it) and never neither."""
import numpy as np
import pytest
import torch

import gpugraphs as G
from gpugraphs import generators as gen

pytestmark = pytest.mark.gpu
N = (1 << 20) - 3


@pytest.fixture(scope="module")
def matrices():
    A = gen.erdos_renyi(N, 16, seed=3)
    I = G.SparseGPUMatrixCSR(N, N, A.rowptr, A.colval, (A.nzval * 255).to(torch.int32) + 1)
    return {"f32": A, "i32": I, "f32 sell": G.SparseGPUMatrixSELL(A, 32, 64),
            "i32 sell": G.SparseGPUMatrixSELL(I, 32, 64)}


@pytest.mark.parametrize("k", [4, 33])
@pytest.mark.parametrize("name", ["f32", "f32 sell", "i32", "i32 sell"])
def test_masks_select_rows_of_the_whole_product(matrices, name, k):
    A = matrices[name]
    g = torch.Generator(device="cuda").manual_seed(k)
    if name.startswith("f32"):
        B, op = torch.rand(k, N, generator=g, device="cuda").T, {}
    else:
        B = torch.randint(0, 1000, (k, N), generator=g, device="cuda", dtype=torch.int32).T
        op = dict(mul=G.GPUGraphs_mul, add=G.GPUGraphs_min, accum=G.GPUGraphs_add)
    C0 = torch.randint(0, 9, (k, N), generator=g, device="cuda").to(B.dtype).T
    whole = C0.clone(memory_format=torch.preserve_format)
    G.gpu_spmm_(whole, A, B, **op)
    rows = torch.rand(N, generator=g, device="cuda")
    for kept in (0.0, 1e-5, 0.003, 0.02, 0.3, 1.0):
        for dtype in (torch.bool, torch.float32):
            mask = (rows < kept).to(dtype)
            C = C0.clone(memory_format=torch.preserve_format)
            G.gpu_spmm_(C, A, B, mask=mask, **op)
            assert torch.equal(C, torch.where((mask != 0)[:, None], whole, C0))


def test_masked_hub_rows():
    """Rows of many pieces, kept and not, on either side of the choice."""
    r = np.random.default_rng(2)
    deg = r.integers(1, 4, N)
    deg[[5, N // 2]] = 40000
    rp = np.concatenate([[1], 1 + np.cumsum(deg)]).astype(np.int32)
    cv = r.integers(1, N + 1, rp[-1] - 1).astype(np.int32)
    A = G.SparseGPUMatrixCSR(N, N, rp, cv, r.integers(1, 9, len(cv)).astype(np.int32))
    B = torch.randint(0, 1000, (8, N), device="cuda", dtype=torch.int32).T
    whole = torch.zeros(8, N, device="cuda", dtype=torch.int32).T
    G.gpu_spmm_(whole, A, B)
    for rows in ([5], [6], [5, N // 2, N - 1], slice(0, N, 2), slice(4, N // 2)):
        mask = torch.zeros(N, dtype=torch.bool, device="cuda")
        mask[rows] = True
        C = torch.full((8, N), 7, device="cuda", dtype=torch.int32).T
        G.gpu_spmm_(C, A, B, mask=mask)
        assert torch.equal(C, torch.where(mask[:, None], whole, torch.full_like(whole, 7)))
