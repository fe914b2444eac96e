"""SCC by contraction (contract_device.cuh): the path that sparse graphs
without hubs take in the cooperative kernel by default.  Labels must equal the
oracle's, and the colour rounds' (colour_mode 0, which never contracts), on
graphs that contract fully, that finish in the one-block tail, that leave a
core to the searches, and that are turned away."""
from __future__ import annotations

import numpy as np
import pytest

import connectivity_gb300 as gb
import oracle
from tests import graphs

pytestmark = pytest.mark.gpu

STARTED = 20  # trace mode of a contraction's start


def _perm(n, s, d, seed):
    p = np.random.default_rng(seed).permutation(n).astype(np.int32)
    return n, p[s], p[d]


def _one_way(k):
    """k x k streets, one way in turn: every vertex has two ways in and out,
    so nothing but the border contracts and the core is left to the searches."""
    v = np.arange(k * k, dtype=np.int32).reshape(k, k)
    s = [v[0::2, :-1], v[1::2, 1:], v[:-1, 0::2], v[1:, 1::2]]
    d = [v[0::2, 1:], v[1::2, :-1], v[1:, 0::2], v[:-1, 1::2]]
    return (k * k, np.concatenate([x.ravel() for x in s]), np.concatenate([x.ravel() for x in d]))


def _two_way(k):
    v = np.arange(k * k, dtype=np.int32).reshape(k, k)
    a = np.concatenate([v[:, :-1].ravel(), v[:-1].ravel()])
    b = np.concatenate([v[:, 1:].ravel(), v[1:].ravel()])
    return k * k, np.concatenate([a, b]), np.concatenate([b, a])


def _cases():
    out = [("grid_33", graphs.grid(33)), ("grid_200", graphs.grid(200)),
           ("grid_perm", _perm(*graphs.grid(150), 1)), ("one_way_31", _one_way(31)),
           ("one_way_200", _one_way(200)), ("two_way_100", _two_way(100)),
           ("cycle_perm", _perm(*graphs.cycle(50000), 2)), ("cycle_long", graphs.cycle(200000)),
           ("path_long", graphs.path(100001))]
    for n in (1023, 1025, 30000):  # around the tail's vertex bound, and above
        for f in (1.2, 2.0, 3.5):
            out.append((f"random_{n}_{f}", graphs.erdos(n, int(n * f), n)))
    return out


CASES = _cases()


@pytest.mark.parametrize("name,case", CASES, ids=[c[0] for c in CASES])
@pytest.mark.parametrize("kw", [{}, {"trim_level": 0}, {"trim_level": 2, "grid_blocks": 5}],
                         ids=["default", "trim0", "trim2_5blocks"])
def test_labels_equal(ctx, name, case, kw):
    n, s, d = case
    g = gb.Graph.from_edges(ctx, n, s, d)
    lab, st = ctx.scc(g, o=gb.opts(small_path=0, **kw), stats=True)
    assert st.unassigned == 0
    trace = [r[2] for r in ctx.reach_trace()]
    if st.n_trim < n and len(trace) < 128:  # (the trace keeps its last 128 records)
        assert STARTED in trace
    assert np.array_equal(lab, oracle.scc(oracle.CpuGraph(n, s, d)))
    if n <= 40000:
        assert np.array_equal(ctx.scc(g, o=gb.opts(small_path=0, colour_mode=0)), lab)
    g.close()


def test_hubs_are_turned_away(ctx):
    """A valid vertex with more than 32 edges on one side keeps the searches,
    whether or not it is the pivot."""
    n, s, d = graphs.grid(64)
    hub = np.full(40, 5, np.int32)
    far = np.arange(100, 140, dtype=np.int32)
    for a, b in ((hub, far), (far, hub)):
        # (and a two-cycle, so that the trim leaves the hub valid)
        s2, d2 = np.r_[s, a, [5, 6]].astype(np.int32), np.r_[d, b, [6, 5]].astype(np.int32)
        g = gb.Graph.from_edges(ctx, n, s2, d2)
        lab = ctx.scc(g, o=gb.opts(small_path=0))
        assert 22 not in [r[2] for r in ctx.reach_trace()]  # no round ran
        assert np.array_equal(lab, oracle.scc(oracle.CpuGraph(n, s2, d2)))
        g.close()


def test_options_that_keep_the_reference_phases(ctx):
    """colour_mode 0 and 1, further FW-BW rounds and labels as the phases
    make them never contract."""
    n, s, d = graphs.grid(64)
    g = gb.Graph.from_edges(ctx, n, s, d)
    for kw in ({"colour_mode": 0}, {"colour_mode": 1}, {"fwbw_rounds": 2}, {"canonical": 0},
               {"expand_mode": 1}):
        ctx.scc(g, o=gb.opts(small_path=0, **kw))
        assert STARTED not in [r[2] for r in ctx.reach_trace()]
    g.close()
