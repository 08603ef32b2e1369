"""SpMM over row ranges of column-major and odd-width operands: short ranges take B where it
lies, long ones through row-major scratch (two launches more), and either writes the range
alone.  Rows fold in storage order up to 256 entries, so the ranges of one matrix agree with
the whole product bit for bit."""
import numpy as np
import pytest
import torch

import gpugraphs as G
from gpugraphs import generators as gen
from gpugraphs.tracing import launch_trace

pytestmark = pytest.mark.gpu


def operands(n, k, layout, dtype):
    g = torch.Generator(device="cuda").manual_seed(k)
    if dtype == torch.int32:
        B = torch.randint(0, 1000, (n, k), generator=g, device="cuda", dtype=dtype)
    else:
        B = torch.rand(n, k, generator=g, device="cuda")
    C = torch.randint(0, 9, (n, k), generator=g, device="cuda").to(dtype)
    return (B, C) if layout == "row" else (B.T.contiguous().T, C.T.contiguous().T)


@pytest.mark.parametrize("layout,k,dtype,short,long", [
    ("col", 5, torch.float32, 1000, 100000), ("col", 33, torch.float32, 500, 20000),
    ("row", 7, torch.float32, 100000, 400000), ("row", 31, torch.float32, 100000, 400000),
    ("col", 32, torch.int32, 10000, 100000), ("col", 3, torch.int32, 100000, 700000)])
@pytest.mark.parametrize("sell", [False, True])
def test_ranges_equal_the_whole_product(layout, k, dtype, short, long, sell):
    n = (1 << 20) - 3
    A = gen.erdos_renyi(n, 16, seed=3)
    if dtype == torch.int32:
        A = G.SparseGPUMatrixCSR(n, n, A.rowptr, A.colval, (A.nzval * 255).to(dtype) + 1)
        op = dict(mul=G.GPUGraphs_safe_add, add=G.GPUGraphs_min, accum=G.GPUGraphs_min)
    else:
        op = {}
    if sell:
        A = G.SparseGPUMatrixSELL(A, 32, 64)
    B, C0 = operands(n, k, layout, dtype)
    whole = C0.clone(memory_format=torch.preserve_format)
    G.gpu_spmm_(whole, A, B, **op)
    launches = {}
    for rows in (1, short, long, n):
        for lo in {1, n // 3, n - rows + 1}:
            if lo + rows - 1 > n or lo < 1:
                continue
            C = C0.clone(memory_format=torch.preserve_format)
            with launch_trace() as t:
                G.gpu_spmm_(C, A, B, range=(lo, lo + rows - 1), **op)
            launches.setdefault(rows, set()).add(t.launches)
            ref = C0.clone(memory_format=torch.preserve_format)
            ref[lo - 1:lo - 1 + rows] = whole[lo - 1:lo - 1 + rows]
            assert torch.equal(C, ref)
    staged = 1 if dtype == torch.int32 else 2
    if layout == "col" or not sell:
        assert min(launches[long]) == min(launches[n]) >= max(launches[short]) + staged
        assert launches[1] == launches[short]


def test_range_beside_and_over_a_hub():
    """A row of many pieces makes rewriting B pay for a few rows already."""
    n = 1 << 17
    rng = np.random.default_rng(2)
    deg = rng.integers(1, 9, n)
    deg[5000] = 40000
    rp = np.concatenate([[1], 1 + np.cumsum(deg)]).astype(np.int32)
    cv = rng.integers(1, n + 1, rp[-1] - 1).astype(np.int32)
    A = G.SparseGPUMatrixCSR(n, n, rp, cv, rng.random(len(cv), dtype=np.float32))
    B, C0 = operands(n, 4, "col", torch.float32)
    whole = C0.clone(memory_format=torch.preserve_format)
    G.gpu_spmm_(whole, A, B)
    count = {}
    for lo, hi in ((4001, 4030), (4970, 5030), (5001, 5001), (5033, 5064)):
        C = C0.clone(memory_format=torch.preserve_format)
        with launch_trace() as t:
            G.gpu_spmm_(C, A, B, range=(lo, hi))
        count[lo] = t.launches
        assert torch.equal(C[:lo - 1], C0[:lo - 1]) and torch.equal(C[hi:], C0[hi:])
        torch.testing.assert_close(C[lo - 1:hi], whole[lo - 1:hi], rtol=1e-5, atol=1e-5)
    assert count[4970] == count[5001] > count[4001] == count[5033]


@pytest.mark.parametrize("k", [4, 33])
def test_masks_of_few_rows(k):
    """Tiles of the staged result without a kept row are left out."""
    n = 70001
    A = gen.erdos_renyi(n, 16, seed=4)
    B, C0 = operands(n, k, "col", torch.float32)
    whole = C0.clone(memory_format=torch.preserve_format)
    G.gpu_spmm_(whole, A, B)
    for rows in ([], [0], [31, 32, 69999, 70000], list(range(0, n, 997))):
        mask = torch.zeros(n, dtype=torch.bool, device="cuda")
        mask[rows] = True
        C = C0.clone(memory_format=torch.preserve_format)
        G.gpu_spmm_(C, A, B, mask=mask)
        assert torch.equal(C, torch.where(mask[:, None], whole, C0))
