"""One-block SCC of graphs with a hub, and host edge lists around the length
up to which the block reads them in place, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import connectivity_gb300 as gb
from tests import graphs
from tests.test_gpu_small import MAX_N, _check_all, _want

pytestmark = pytest.mark.gpu


def _with_hub(n, s, d, hub, k, seed):
    """k edges from and to `hub`, on top of a graph."""
    r = np.random.default_rng(seed)
    far = r.integers(0, n, 2 * k).astype(np.int32)
    h = np.full(k, hub, np.int32)
    return n, np.r_[s, h, far[k:]].astype(np.int32), np.r_[d, far[:k], h].astype(np.int32)


@pytest.mark.parametrize("k", [15, 16, 400])  # around the degree that makes a hub
@pytest.mark.parametrize("what", ["sparse", "grid", "path_out", "path_back", "dense"])
def test_hub_path(ctx, k, what):
    """Graphs with a hub (searches from below, contraction of the rest): a
    rest of many components, a rest larger than the contraction takes, long
    chains in and out of the hub's component, lists longer than a lane's share."""
    if what == "sparse":
        n, s, d = graphs.erdos(MAX_N, MAX_N, 21)
    elif what == "grid":
        n, s, d = graphs.grid(60)
    elif what == "dense":
        n, s, d = graphs.erdos(300, 12000, 22)
    else:
        n, s, d = graphs.path(3000)
        if what == "path_back":
            s, d = np.r_[s, n - 1].astype(np.int32), np.r_[d, 7].astype(np.int32)
    n, s, d = _with_hub(n, s, d, n // 3, k, k)
    _check_all(ctx, "scc", n, s, d)
    p = np.random.default_rng(k).permutation(n).astype(np.int32)
    _check_all(ctx, "scc", n, p[s], p[d])


@pytest.mark.parametrize("kind", ["scc", "wcc"])
@pytest.mark.parametrize("m", [1, 8191, 8193, 65536, 65537])
def test_host_list_lengths(ctx, kind, m):
    """The longest list read in place and the first that is copied; an id
    outside [0, n) in the last edge is refused in both."""
    n = 5000
    r = np.random.default_rng(m)
    s, d = r.integers(0, n, (2, m)).astype(np.int32)
    run = ctx.scc_edges if kind == "scc" else ctx.wcc_edges
    want = _want(kind, n, s, d)
    assert np.array_equal(run(n, s, d), want)
    d[-1] = n
    with pytest.raises(gb.GBError):
        run(n, s, d)
    d[-1] = 0
    assert np.array_equal(run(n, s, d), _want(kind, n, s, d))
