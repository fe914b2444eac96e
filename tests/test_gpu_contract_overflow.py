"""Contractions and residuals whose arrays run out: the round that overflowed
is open, the searches and colour rounds label what it merged, and the labels
are the oracle's.  Each on a context of its own and again after a larger graph
has run there."""
from __future__ import annotations

import numpy as np
import pytest

import connectivity_gb300 as gb
import oracle
from tests import graphs

pytestmark = pytest.mark.gpu


def _fork(k, f, base=0):
    """k copies of u <-> y, u -> v, u -> w, v -> z and w -> z (f edges each),
    z -> p, p <-> q.  An IN1 round hooks v and w onto u and logs their 2 f
    edges to z, the OUT1 round after it hooks z onto p, logs the same 2 f
    edges again and leaves no vertex alive."""
    u, y, v, w, z, p, q = (base + i * k + np.arange(k) for i in range(7))
    s = np.r_[u, y, u, u, np.repeat(v, f), np.repeat(w, f), z, p, q]
    d = np.r_[y, u, v, w, np.repeat(z, f), np.repeat(z, f), p, q, p]
    return base + 7 * k, s.astype(np.int32), d.astype(np.int32)


def _ring(k, f, base=0):
    """k copies of a component that drops a fifth of its edges in the first
    round and hardly any in the second: u <-> y, u -> v, u -> w, v -> z and
    w -> z (f edges each), z -> p and z -> r, p <-> q, r <-> t, p -> u, r -> u."""
    u, y, v, w, z, p, q, r, t = (base + i * k + np.arange(k) for i in range(9))
    s = np.r_[u, y, u, u, np.repeat(v, f), np.repeat(w, f), z, z, p, q, r, t, p, r]
    d = np.r_[y, u, v, w, np.repeat(z, f), np.repeat(z, f), p, r, q, p, t, r, u, u]
    return base + 9 * k, s.astype(np.int32), d.astype(np.int32)


def _join(n, s, d, add):
    n2, s2, d2 = add(n)
    return n2, np.r_[s, s2].astype(np.int32), np.r_[d, d2].astype(np.int32)


def _shuffle(n, s, d, seed):
    p = np.random.default_rng(seed).permutation(n).astype(np.int32)
    return n, p[s], p[d]


def _cores(n, m):
    """Two components of random edges with a hub each: the search takes one,
    the other one's edges exceed the residual's list of n pairs."""
    _, s, d = graphs.erdos(n, m, 1)
    h = np.arange(64, dtype=np.int32)
    s, d = np.r_[s, np.zeros(64, np.int32), h], np.r_[d, h, np.zeros(64, np.int32)]
    return 2 * n, np.r_[s, s + n].astype(np.int32), np.r_[d, d + n].astype(np.int32)


CASES = {
    # 60,000 logged edges of a graph of 40,500, and no vertex alive after them
    "log_and_empty": _fork(1500, 10),
    "log_shuffled": _shuffle(*_fork(1500, 10), 3),
    # beside a lattice, which keeps vertices alive
    "log_and_grid": _join(*graphs.grid(40), lambda b: _fork(1500, 10, b)),
    # 48,000 and 45,000 edges in the first two rounds for 60,000 places
    "edges": _ring(1500, 14),
    "edges_shuffled": _shuffle(*_ring(1500, 14), 4),
    # a residual that the one-block tail takes, whose log of 2,560 gets 4,400
    "tail_log": _join(*gb.rmat_edges(14, 16, 3), lambda b: _fork(55, 20, b)),
    # a residual of more edges than its list
    "residual_list": _cores(20000, 600000),
}


@pytest.mark.parametrize("name", CASES)
def test_labels_equal(name):
    n, s, d = CASES[name]
    want = oracle.scc(oracle.CpuGraph(n, s, d))
    ctx = gb.Context(0)
    g = gb.Graph.from_edges(ctx, n, s, d)
    assert np.array_equal(ctx.scc(g, o=gb.opts(small_path=0)), want)
    big = gb.Graph.from_edges(ctx, *graphs.grid(600))
    ctx.scc(big)
    assert np.array_equal(ctx.scc(g, o=gb.opts(small_path=0)), want)
    assert np.array_equal(ctx.scc(g, o=gb.opts(small_path=0, colour_mode=0)), want)
    g.close()
    big.close()
    ctx.close()


@pytest.mark.parametrize("seed", [0, 1])
def test_one_block_log(ctx, seed):
    """A one-block graph with a hub, whose rest logs 2,304 edges for 1,280 places."""
    n, s, d = graphs.erdos(600, 3000, 5)
    h = np.arange(40, dtype=np.int32)
    s, d = np.r_[s, np.zeros(40, np.int32), h], np.r_[d, h, np.zeros(40, np.int32)]
    n, s, d = _join(n, s, d, lambda b: _fork(36, 16, b))
    if seed:
        n, s, d = _shuffle(n, s, d, seed)
    g = gb.Graph.from_edges(ctx, n, s, d)
    want = oracle.scc(oracle.CpuGraph(n, s, d))
    assert np.array_equal(ctx.scc(g, o=gb.opts(small_path=2)), want)
    assert np.array_equal(ctx.scc_edges(n, s, d), want)
    g.close()
