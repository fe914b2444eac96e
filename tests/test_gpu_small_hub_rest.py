"""One-block SCC of graphs with a hub whose searches are given up, or leave
more than the contraction takes: the general way's trim and rounds label the
rest, in as many steps as without a hub, and the labels are the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import connectivity_gb300 as gb
import oracle
from tests import graphs

pytestmark = pytest.mark.gpu


def _hub_and_chain(core, chain, how):
    """A random core with a hub of 40 edges each way, and a chain: out of the
    core, into it, apart from it, or apart with a two-cycle at both ends."""
    n, s, d = graphs.erdos(core, 4 * core, core)
    far = np.random.default_rng(chain).integers(0, core, 80)
    c = core + np.arange(chain)
    s = np.r_[s, np.zeros(40, np.int64), far[40:], c[:-1]]
    d = np.r_[d, far[:40], np.zeros(40, np.int64), c[1:]]
    ends = {"out": ([1], [c[0]]), "in": ([c[-1]], [1]), "apart": ([], []),
            "loops": ([c[1], c[-1]], [c[0], c[-2]])}[how]
    return core + chain, np.r_[s, ends[0]].astype(np.int32), np.r_[d, ends[1]].astype(np.int32)


# around the work after which the searches stop (32 passes up to 1,024
# vertices, 16 up to 2,048, 8 from 4,097), and around the 512 vertices that the
# contraction takes
@pytest.mark.parametrize("core,chain", [(500, 31), (500, 33), (512, 512), (513, 512), (500, 513),
                                        (300, 700), (1500, 15), (1500, 17), (1500, 548),
                                        (1500, 600), (5000, 7), (5000, 9), (5000, 1144)])
@pytest.mark.parametrize("how", ["out", "in", "apart", "loops"])
def test_labels_equal(ctx, core, chain, how):
    n, s, d = _hub_and_chain(core, chain, how)
    want = oracle.scc(oracle.CpuGraph(n, s, d))
    g = gb.Graph.from_edges(ctx, n, s, d)
    assert np.array_equal(ctx.scc(g, o=gb.opts(small_path=2)), want)
    assert np.array_equal(ctx.scc_edges(n, s, d), want)
    g.close()


def test_a_chain_is_trimmed_from_both_ends(ctx):
    """1,500 steps for a chain of 3,000 beside the hub's component.  Without
    the trim a colour would walk down the whole chain."""
    n, s, d = _hub_and_chain(600, 3000, "apart")
    g = gb.Graph.from_edges(ctx, n, s, d)
    lab = ctx.scc(g, o=gb.opts(small_path=2, max_steps=1700))
    assert np.array_equal(lab, oracle.scc(oracle.CpuGraph(n, s, d)))
    g.close()
