"""The rounds of a contraction that the statistics report do not vary from run
to run, although the order of its lists does."""
from __future__ import annotations

import numpy as np
import pytest

import connectivity_gb300 as gb
from tests import graphs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [graphs.path(20001), graphs.cycle(9000), graphs.grid(150)],
                         ids=["path", "cycle", "grid"])
def test_rounds_repeat(ctx, case):
    g = gb.Graph.from_edges(ctx, *case)
    rounds = {ctx.scc(g, np.empty(g.n, np.int32), gb.opts(small_path=0), stats=True)[1].colour_rounds
              for _ in range(100)}
    assert len(rounds) == 1, rounds
    g.close()
