"""What the searches leave of an SCC run: rests around the size up to which the
residual phase looks at them, and one whose edges exceed its list."""
from __future__ import annotations

import numpy as np
import pytest

import connectivity_gb300 as gb
import oracle

pytestmark = pytest.mark.gpu


def _star_and_tree(k, extra):
    """A two-way star of 1,000 leaves, whose centre is the pivot, and apart from
    it a two-way random tree of k vertices, which is left whole; `extra` one-way
    edges lead from the star into vertices that lead back to the tree's root."""
    r = np.random.default_rng(k)
    leaf = np.arange(1, 1001)
    v = 1001 + np.arange(1, k)
    up = 1001 + (r.random(k - 1) * np.arange(1, k)).astype(np.int64)
    x = 1001 + k + np.arange(extra)
    s = np.r_[np.zeros(1000, np.int64), leaf, up, v, leaf[:extra], x]
    d = np.r_[leaf, np.zeros(1000, np.int64), v, up, x, np.full(extra, 1001)]
    return 1001 + k + extra, s.astype(np.int32), d.astype(np.int32)


# 2^18 vertices left, one less and one more; 131,072 edges listed, and more
@pytest.mark.parametrize("k", [65536, 65537, (1 << 18) - 101, (1 << 18) - 100, (1 << 18) - 99])
def test_labels_equal(ctx, k):
    n, s, d = _star_and_tree(k, 100)
    g = gb.Graph.from_edges(ctx, n, s, d)
    want = oracle.scc(oracle.CpuGraph(n, s, d))
    assert np.array_equal(ctx.scc(g), want)
    assert np.array_equal(ctx.scc(g, o=gb.opts(colour_mode=0)), want)
    assert np.array_equal(ctx.scc_edges(n, s, d), want)
    g.close()
