"""Padded SELL handles whose values change: the sorted copy pays after some eight products, so
values that do not last take the handle's own slices (one launch, or two with chunks, where
the copy's relabelled columns take one more)."""
import pytest
import torch

import gpugraphs as G
from gpugraphs import core
from gpugraphs import generators as gen
from gpugraphs.tracing import launch_trace

pytestmark = pytest.mark.gpu


def changed(A):
    core.check(core.lib().gg_mat_values_changed(core.ctx(), A.handle), core.lib())


@pytest.mark.parametrize("C", [8, 32])
def test_copy_follows_how_long_values_last(C):
    A = gen.rmat(21, 16, seed=3, wkind=gen.W_INT_1_255)  # columns enough for the relabelling
    S = G.SparseGPUMatrixSELL(A, C, 64)
    x = torch.randint(0, 5000, (A.n,), device="cuda", dtype=torch.int32)
    op = dict(mul=G.GPUGraphs_safe_add, add=G.GPUGraphs_min)
    ref = torch.zeros_like(x)
    G.gpu_spmv_(ref, A, x, **op)

    def launches(products):
        for _ in range(products):
            y = torch.zeros_like(x)
            with launch_trace() as t:
                G.gpu_spmv_(y, S, x, **op)
            assert torch.equal(y, ref)
        return t.launches
    copy = launches(1)  # a first product makes the copy
    assert copy == 3
    for _ in range(2):  # one product for each set of values: none
        changed(S)
        assert launches(1) == 2
    changed(S)
    changed(S)  # several entries written before the next product
    assert launches(8) == 2
    changed(S)
    assert launches(7) == copy  # the last values were used eight times
    changed(S)
    assert launches(1) == 2


def test_new_values_reach_either_layout():
    A = gen.rmat(16, 16, seed=4, wkind=gen.W_INT_1_255)
    S = G.SparseGPUMatrixSELL(A, 32, 64)
    x = torch.randint(0, 5000, (A.n,), device="cuda", dtype=torch.int32)
    op = dict(mul=G.GPUGraphs_safe_add, add=G.GPUGraphs_min)
    for products in (1, 1, 9, 1, 1):
        A.nzval.add_(3)
        S.nzval[S.colval > 0] += 3
        A.values_changed()
        changed(S)
        ref, y = torch.zeros_like(x), torch.zeros_like(x)
        G.gpu_spmv_(ref, A, x, **op)
        for _ in range(products):
            G.gpu_spmv_(y, S, x, **op)
            assert torch.equal(y, ref)
