"""Tuned choices and the kernels that then run: what another handle gets from a choice, and
what the order of calls must not change.  Kernels are told apart by their launch counts."""
import numpy as np
import pytest
import torch

import gpugraphs as G
from gpugraphs import generators as gen
from gpugraphs import tuning
from gpugraphs.tracing import launch_trace

pytestmark = pytest.mark.gpu


def product(A, x):
    """(launches, result) of a Float32 plus-times product; the first call builds its layout."""
    y = torch.zeros(A.m, dtype=torch.float32, device="cuda")
    G.gpu_spmv_(y, A, x)
    with launch_trace() as t:
        G.gpu_spmv_(y, A, x)
    return t.launches, y


@pytest.mark.parametrize("sigma", [0, 64])
def test_applied_choice_runs_the_kernel_that_was_timed(sigma):
    """On a CSR handle and on a padded SELL handle, whose sorted copy a choice must not bar."""
    def handle():
        A = gen.rmat(20 if sigma == 0 else 18, 16, seed=9, wkind=gen.W_U01_F32)
        return G.SparseGPUMatrixSELL(A, 32, sigma) if sigma else A
    A, B = handle(), handle()
    x = torch.rand(A.n, device="cuda")
    res = tuning.autotune(A)
    tuning.apply(B, res)
    (la, ya), (lb, yb) = product(A, x), product(B, x)
    assert la == lb and torch.equal(ya, yb)


@pytest.mark.parametrize("sigma", [0, 64])
def test_built_in_choice_undoes_a_tuned_one(sigma):
    A = gen.rmat(18, 16, seed=9, wkind=gen.W_U01_F32)
    if sigma:
        A = G.SparseGPUMatrixSELL(A, 32, sigma)
    x = torch.rand(A.n, device="cuda")
    la, ya = product(A, x)
    tuning.apply(A, {"spmv_kernel": "sell", "slice_size": 32, "sigma": sigma or A.m,
                     "sell_variant": "bulk_copy", "hot_cols": 16384})
    assert product(A, x)[0] != la
    tuning.apply(A, {"spmv_kernel": "sell", "slice_size": 32, "sigma": sigma or A.m,
                     "sell_variant": "built_in"})
    lb, yb = product(A, x)
    assert la == lb and torch.equal(ya, yb)


@pytest.mark.parametrize("first", ["plain", "masked", "minplus", "spmm1"])
def test_choice_outlives_whichever_product_comes_first(first):
    """A kernel chosen before the copy exists runs, whatever product makes the copy."""
    A = gen.rmat(17, 16, seed=9, wkind=gen.W_U01_F32)
    x = torch.rand(A.n, device="cuda")
    built_in, _ = product(A, x)
    B = gen.rmat(17, 16, seed=9, wkind=gen.W_U01_F32)
    tuning.apply(B, {"sell_variant": "bulk_copy"})
    y = torch.zeros(B.m, device="cuda")
    if first == "masked":
        G.gpu_spmv_(y, B, x, mask=torch.ones(B.m, dtype=torch.bool, device="cuda"))
    elif first == "minplus":
        G.gpu_spmv_(y, B, x, mul=G.GPUGraphs_safe_add, add=G.GPUGraphs_min)
    elif first == "spmm1":
        G.gpu_spmm_(y.view(-1, 1), B, x.view(-1, 1))
    tuned, yb = product(B, x)
    C = gen.rmat(17, 16, seed=9, wkind=gen.W_U01_F32)
    tuning.apply(C, {"sell_variant": "bulk_copy"})
    ref, yc = product(C, x)
    assert tuned == ref != built_in and torch.equal(yb, yc)


@pytest.mark.parametrize("m", [3000, 65535, 65536])
def test_chosen_copy_runs_at_every_size(m):
    """A SELL-32 layout chosen for a matrix below 65536 rows: a hub's row comes in chunks of
    128 entries, folded by a second launch that row blocks do not make."""
    rng = np.random.default_rng(m)
    deg = rng.integers(1, 9, m)
    deg[7] = 2000
    rp = np.concatenate([[1], 1 + np.cumsum(deg)]).astype(np.int32)
    cv = rng.integers(1, m + 1, rp[-1] - 1).astype(np.int32)
    nz = rng.random(len(cv), dtype=np.float32)
    A = G.SparseGPUMatrixCSR(m, m, rp, cv, nz)
    tuning.apply(A, {"spmv_kernel": "sell", "slice_size": 32, "sigma": m})
    x = torch.rand(m, device="cuda")
    launches, y = product(A, x)
    assert launches == 2 and G.spmv_layout(A) == "sell"
    ref = np.add.reduceat(nz.astype(np.float64) * x.cpu().numpy()[cv - 1], rp[:-1] - 1)
    np.testing.assert_allclose(y.cpu().numpy(), ref, rtol=1e-5)
