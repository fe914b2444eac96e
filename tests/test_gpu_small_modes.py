"""One-block SCC of device graphs in every colour mode, graphs of other sizes
in turn: the block's offsets are complete before another thread reads them."""
from __future__ import annotations

import numpy as np
import pytest

import connectivity_gb300 as gb
import oracle
from tests import graphs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_labels_in_turn(ctx, mode):
    cases = [graphs.erdos(6144, 9000, 1), graphs.path(3000), graphs.erdos(1023, 8000, 2),
             graphs.cycle(4097), graphs.grid(60)]
    gs = [(gb.Graph.from_edges(ctx, *c), oracle.scc(oracle.CpuGraph(*c))) for c in cases]
    o = gb.opts(small_path=2, colour_mode=mode)
    for _ in range(10):
        for g, want in gs:
            assert np.array_equal(ctx.scc(g, o=o), want)
    for g, _ in gs:
        g.close()
