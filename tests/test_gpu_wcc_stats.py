"""Statistics of a WCC run: the phases that they describe are run for a caller
who asks for them, also on a graph that takes the union-find otherwise."""
from __future__ import annotations

import numpy as np
import pytest

import connectivity_gb300 as gb
import oracle
from tests import graphs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [graphs.grid(120), graphs.erdos(20000, 24000, 3)],
                         ids=["grid", "random"])
def test_counts_of_a_sparse_graph(ctx, case):
    n, s, d = case
    g = gb.Graph.from_edges(ctx, n, s, d)
    lab, st = ctx.wcc(g, stats=True)
    want = oracle.cc(oracle.CpuGraph(n, s, d, mirror=True))
    assert np.array_equal(lab, want) and np.array_equal(ctx.wcc(g), want)
    deg = np.bincount(s, minlength=n) + np.bincount(d, minlength=n)
    assert st.pivot == int(np.argmax(deg))
    assert st.n_visit_fw == int((want == want[st.pivot]).sum())
    assert st.fw_steps > 0 and st.unassigned == 0
    g.close()
