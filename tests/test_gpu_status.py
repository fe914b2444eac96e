"""Status of runs on the one-block and the cooperative path: the kernels keep
the error latch themselves."""
from __future__ import annotations

import numpy as np
import pytest

import connectivity_gb300 as gb
import oracle
from tests import graphs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("small", [0, 2])
def test_latch(ctx, small):
    """A later good asynchronous run leaves the latched error, a sync reports
    and clears it, and a run that the host waits for clears it too; a failed
    waited run is reported by itself and leaves nothing behind."""
    torch = pytest.importorskip("torch")
    n, s, d = graphs.grid(40)
    g = gb.Graph.from_edges(ctx, n, s, d)
    lab = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    bad, good = gb.opts(max_steps=1, small_path=small), gb.opts(small_path=small)
    want = oracle.scc(oracle.CpuGraph(n, s, d))
    ctx.sync()
    ctx.scc_async(g, lab.data_ptr(), bad)
    ctx.scc_async(g, lab.data_ptr(), good)
    with pytest.raises(gb.GBError):
        ctx.sync()
    ctx.sync()
    assert np.array_equal(lab.cpu().numpy(), want)
    ctx.scc_async(g, lab.data_ptr(), bad)
    assert np.array_equal(ctx.scc(g, o=good), want)
    ctx.sync()
    with pytest.raises(gb.GBError):
        ctx.scc(g, o=bad)
    ctx.sync()
    assert np.array_equal(ctx.scc(g, o=good), want)
    g.close()
