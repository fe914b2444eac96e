"""Step caps: a cap that the searches and rounds could meet keeps them, so that
it stops the calls that it always stopped.  The shorter ways (contraction,
residual phase, union-find, one-block searches from a hub) count other steps."""
from __future__ import annotations

import numpy as np
import pytest

import connectivity_gb300 as gb
import oracle
from tests import graphs
from tests.test_gpu_small_hub_rest import _hub_and_chain

pytestmark = pytest.mark.gpu

SHORTER = {20, 22, 28}  # trace modes: contraction, its rounds, residual


def _status(call):
    try:
        call()
    except gb.GBError as e:
        return e.status
    return 0


def test_a_long_path_is_still_stopped(ctx):
    """A search down 10,000 vertices takes over 100 steps, whatever they do."""
    n, s, d = graphs.path(10000)
    g = gb.Graph.from_edges(ctx, n, s, d)
    o = gb.opts(max_steps=100)
    for call in (lambda: ctx.wcc(g, o=o), lambda: ctx.wcc_edges(n, s, d, o=o),
                 lambda: ctx.scc(g, o=o), lambda: ctx.scc_edges(n, s, d, o=o)):
        assert _status(call) == 5  # GB_ERR_ITER_LIMIT
    o = gb.opts(max_steps=2 * n + 4096)  # out of their reach: the shorter ways
    assert np.array_equal(ctx.wcc(g, o=o), np.zeros(n))
    assert np.array_equal(ctx.scc(g, o=o), np.arange(n))
    g.close()


@pytest.mark.parametrize("case", [graphs.grid(120), graphs.erdos(20000, 40000, 1),
                                  gb.rmat_edges(14, 16, 1)], ids=["grid", "random", "rmat"])
def test_capped_runs_keep_the_phases(ctx, case):
    n, s, d = case
    g = gb.Graph.from_edges(ctx, n, s, d)
    want = oracle.scc(oracle.CpuGraph(n, s, d))
    free = 2 * n + 4096
    assert np.array_equal(ctx.scc(g, o=gb.opts(max_steps=free)), want)
    assert SHORTER & {r[2] for r in ctx.reach_trace()}
    assert np.array_equal(ctx.scc(g, o=gb.opts(max_steps=free - 1)), want)
    assert not SHORTER & {r[2] for r in ctx.reach_trace()}
    g.close()


def test_a_cap_that_the_hub_searches_would_meet(ctx):
    """One block: 120 steps are enough for the trim of a chain of 100 out of
    the hub's component, and for the searches without it."""
    n, s, d = _hub_and_chain(600, 100, "out")
    want = oracle.scc(oracle.CpuGraph(n, s, d))
    g = gb.Graph.from_edges(ctx, n, s, d)
    o = gb.opts(max_steps=120)
    assert np.array_equal(ctx.scc(g, o=o), want)
    assert np.array_equal(ctx.scc_edges(n, s, d, o=o), want)
    g.close()
