"""BFS of hub-free graphs on both sides of the line between persistent and separate levels."""
import numpy as np
import pytest

from test_search_queue_gpu import _check, _graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", [-1, 0, 1])
@pytest.mark.parametrize("n", [2300, 70002])
def test_entries_per_vertex(n, extra):
    """9 n stored entries, one edge less and one more."""
    r = np.concatenate([np.arange(n)] * 4 + [np.arange(n // 2)])
    c = np.concatenate([(np.arange(n) + s) % n for s in (1, 37, 501, 911)] + [(np.arange(n // 2) + 700) % n])
    if extra < 0:
        r, c = r[:extra], c[:extra]
    elif extra > 0:
        r, c = np.append(r, 5), np.append(c, 905)
    rp, cv, nz = _graph(n, r, c, np.int32, seed=3)
    assert len(cv) == 9 * n + 2 * extra
    _check(n, rp, cv, nz, n - 7)
