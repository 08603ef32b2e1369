"""Searches at the lines between the single-CTA rounds, the persistent kernels, the push and
hub rounds and the pull rounds over the sorted copy.  Levels are integers and distances are
exact fixpoints, so every comparison is exact."""
import numpy as np
import pytest

from test_search_queue_gpu import _check, _graph

pytestmark = pytest.mark.gpu


def _grid(h, w):
    v = np.arange(h * w).reshape(h, w)
    return (np.concatenate([v[:, :-1].ravel(), v[:-1].ravel()]),
            np.concatenate([v[:, 1:].ravel(), v[1:].ravel()]))


@pytest.mark.parametrize("dtype", [np.int32, np.float32])
@pytest.mark.parametrize("h,w", [(23, 89), (32, 64), (3, 683), (1, 2048), (2, 1025), (120, 101)])
def test_small_grids(h, w, dtype):
    """2047 to 2050 vertices and a larger one: below and above the persistent kernels' line,
    with eight CTAs and a remainder; (1, 2048) is one path of 2047 levels."""
    r, c = _grid(h, w)
    _check(h * w, *_graph(h * w, r, c, dtype, seed=h), 1)
    _check(h * w, *_graph(h * w, r, c, dtype, seed=w), h * w // 2 + 1)


@pytest.mark.parametrize("extra", [-1, 0, 1])
@pytest.mark.parametrize("n", [2048, 2300, 70001])
def test_entries_per_vertex(n, extra):
    """6 n stored entries, one edge less and one more: both sides of the line between the
    persistent levels and the separate launches."""
    r = np.concatenate([np.arange(n)] * 3)
    c = np.concatenate([(np.arange(n) + s) % n for s in (1, 37, 501)])
    if extra < 0:
        r, c = r[:extra], c[:extra]
    elif extra > 0:
        r, c = np.append(r, 5), np.append(c, 905)
    rp, cv, nz = _graph(n, r, c, np.int32, seed=3)
    assert len(cv) == 6 * n + 2 * extra
    _check(n, rp, cv, nz, n - 7)


@pytest.mark.parametrize("dtype", [np.int32, np.float32])
@pytest.mark.parametrize("deg", [512, 513])
@pytest.mark.parametrize("n", [12287, 12288, 30011])
def test_hubs_of_medium_graphs(n, deg, dtype):
    """Hubs at the line of the copy's pull rounds: its out-degree and the vertex count."""
    rng = np.random.default_rng(n + deg)
    r, c = rng.integers(2, n, 6 * n), rng.integers(2, n, 6 * n)
    keep = r != c
    r = np.concatenate([r[keep], np.full(deg, 1), [0]])
    c = np.concatenate([c[keep], rng.permutation(np.arange(2, n))[:deg], [2]])
    rp, cv, nz = _graph(n, r, c, dtype, seed=deg)
    assert np.diff(rp).max() == deg
    for source in (1, 2, n):
        _check(n, rp, cv, nz, source)
