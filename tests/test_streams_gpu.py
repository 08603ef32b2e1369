"""Asynchronous calls on two streams that share a workspace: the second waits for the first.
The first stream is kept busy before its call, so a call that did not wait would be done
long before it; calls without a shared workspace do overlap."""
import numpy as np
import pytest
import torch

import gpugraphs as G
from gpugraphs import generators as gen

pytestmark = pytest.mark.gpu
BUSY = 100_000_000  # clocks, some 50 ms


def hub_matrix(n, dtype=np.float32):
    """One row of 9000 entries among short ones: folded from partial results."""
    rng = np.random.default_rng(n)
    deg = rng.integers(1, 5, n)
    deg[3] = 9000
    rp = np.concatenate([[1], 1 + np.cumsum(deg)]).astype(np.int32)
    cv = rng.integers(1, n + 1, rp[-1] - 1).astype(np.int32)
    return G.SparseGPUMatrixCSR(n, n, rp, cv, rng.integers(1, 9, len(cv)).astype(dtype))


def vectors(n, dtype, count=2):
    g = torch.Generator(device="cuda").manual_seed(1)
    return [torch.randint(0, 100, (n,), generator=g, device="cuda").to(dtype) for _ in range(count)]


MINPLUS = dict(mul=G.GPUGraphs_safe_add, add=G.GPUGraphs_min)


def spmv_case(name):
    if name == "plain":  # relabelled x and chunks of the copy
        A, dt, op = gen.rmat(17, 16, seed=2), torch.float32, {}
    elif name == "minplus":
        A, dt, op = gen.rmat(17, 16, seed=2, wkind=gen.W_INT_1_255), torch.int32, MINPLUS
    elif name == "masked":
        A, dt = gen.rmat(17, 16, seed=2), torch.float32
        op = dict(mask=torch.ones(A.m, dtype=torch.bool, device="cuda"))
    elif name == "row_blocks":
        A, dt, op = hub_matrix(5000, np.int32), torch.int32, MINPLUS
    else:  # "sell"
        A = G.SparseGPUMatrixSELL(gen.rmat(17, 16, seed=2), 32, 64)
        dt, op = torch.float32, {}
    xs = vectors(A.n, dt)
    return [(lambda y, x=x: G.gpu_spmv_(y, A, x, **op), torch.zeros(A.m, dtype=dt, device="cuda"))
            for x in xs]


def spmm_case(name):
    if name == "partials":
        A, dt, k, col, op = hub_matrix(5000), torch.float32, 32, False, {}
    elif name == "column_major":
        A, dt, k, col, op = gen.erdos_renyi(70000, 16, seed=2), torch.float32, 8, True, {}
    else:  # "minplus"
        A, dt, k, col, op = hub_matrix(70000, np.int32), torch.int32, 32, True, MINPLUS
    out = []
    for x in vectors(A.n * k, dt):
        B, C = x.view(A.n, k), torch.zeros(A.m, k, dtype=dt, device="cuda")
        if col:
            B, C = B.T.contiguous().T, C.T.contiguous().T
        out.append((lambda y, B=B: G.gpu_spmm_(y, A, B, **op), C))
    return out


def run(calls):
    """Both calls alone, then on two streams with the first one's busy: (ordered, right)."""
    refs = []
    for f, y in calls:
        f(y)
        f(y)
        refs.append(y.clone(memory_format=torch.preserve_format))
        y.zero_()
    torch.cuda.synchronize()
    s, t = torch.cuda.Stream(), torch.cuda.Stream()
    first, second = torch.cuda.Event(), torch.cuda.Event()
    with torch.cuda.stream(s):
        torch.cuda._sleep(BUSY)
        calls[0][0](calls[0][1])
        first.record()
    with torch.cuda.stream(t):
        calls[1][0](calls[1][1])
        second.record()
    second.synchronize()
    ordered = first.query()
    torch.cuda.synchronize()
    return ordered, all(torch.equal(y, r) for (_, y), r in zip(calls, refs))


@pytest.mark.parametrize("name", ["plain", "minplus", "masked", "row_blocks", "sell"])
def test_products_of_one_matrix(name):
    for _ in range(2):
        assert run(spmv_case(name)) == (True, True)


@pytest.mark.parametrize("name", ["partials", "column_major", "minplus"])
def test_dense_products_of_one_context(name):
    for _ in range(2):
        assert run(spmm_case(name)) == (True, True)


def test_search_after_a_dense_product():
    """A search takes the scratch arena that a product on another stream still reads."""
    A = gen.rmat(15, 16, seed=2, wkind=gen.W_PATTERN)
    lev = G.bfs_distances(A, 1).clone()
    calls = spmm_case("column_major")
    calls[1] = (lambda y: y.copy_(G.bfs_distances(A, 1)), torch.zeros_like(lev))
    assert run(calls) == (True, True)


def test_products_without_a_workspace_overlap():
    A = gen.erdos_renyi(16384, 16, seed=2)
    calls = [(lambda y, x=x: G.gpu_spmv_(y, A, x), torch.zeros(A.m, device="cuda"))
             for x in vectors(A.n, torch.float32)]
    assert run(calls) == (False, True)


def test_products_of_two_matrices_overlap():
    assert run([spmv_case("plain")[0], spmv_case("minplus")[0]]) == (False, True)


def test_capture_and_replay():
    """Calls under capture record nothing and wait for nothing outside."""
    (f, y), _ = spmv_case("plain")
    f(y)
    ref = y.clone()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        f(y)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        f(y)
    y.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, ref)
    f(y)
    torch.cuda.synchronize()
    assert torch.equal(y, ref)
