"""WCC by union-find (unionfind.cu): sparse device graphs (ranges joined in
shared memory, then across) and edge lists above the one-block size, against
the oracle and the searches of the cooperative kernel."""
from __future__ import annotations

import numpy as np
import pytest

import connectivity_gb300 as gb
import oracle
from tests import graphs

pytestmark = pytest.mark.gpu


def _perm(n, s, d, seed):
    p = np.random.default_rng(seed).permutation(n).astype(np.int32)
    return n, p[s], p[d]


def _hub(n):
    """A hub whose list is walked by a warp, over a sparse random graph."""
    _, s, d = graphs.erdos(n, n, 5)
    far = np.arange(0, n, 3, dtype=np.int32)
    return n, np.r_[s, np.full(far.size, n // 2, np.int32)], np.r_[d, far]


CASES = [("empty", 9000, np.zeros(0, np.int32), np.zeros(0, np.int32)),
         ("grid_200",) + graphs.grid(200), ("grid_perm",) + _perm(*graphs.grid(150), 1),
         ("path",) + graphs.path(1000003), ("path_perm",) + _perm(*graphs.path(200000), 2),
         ("cycle",) + graphs.cycle(65536), ("hub",) + _hub(50000)]
# around the smallest range of a block, and several ranges
CASES += [(f"random_{n}",) + graphs.erdos(n, int(1.1 * n), n) for n in (2047, 2048, 2049, 700001)]


@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_sparse_device_graph(ctx, case):
    _, n, s, d = case
    g = gb.Graph.from_edges(ctx, n, s, d)
    want = oracle.cc(oracle.CpuGraph(n, s, d, mirror=True))
    assert np.array_equal(ctx.wcc(g, o=gb.opts(small_path=0)), want)
    if n <= 100000:  # the searches (further FW-BW rounds keep them) agree
        assert np.array_equal(ctx.wcc(g, o=gb.opts(small_path=0, fwbw_rounds=2)), want)
    g.close()


def test_symmetric_csr(ctx):
    n, s, d = graphs.grid(120)
    a, b = np.r_[s, d], np.r_[d, s]
    off, adj = gb.csr_from_edges(n, a, b)
    g = gb.Graph.from_csr(ctx, n, off, adj)
    assert g.symmetric and g.m < 8 * n
    assert np.array_equal(ctx.cc(g), oracle.cc(oracle.CpuGraph(n, s, d, mirror=True)))
    g.close()


LISTS = [c for c in CASES if c[1] > 6144] + [("rmat_17",) + gb.rmat_edges(17, 16, 3),
                                             ("grid_100",) + graphs.grid(100)]


@pytest.mark.parametrize("case", LISTS, ids=[c[0] for c in LISTS])
@pytest.mark.parametrize("device", [False, True], ids=["host", "device"])
def test_edge_list(ctx, case, device):
    torch = pytest.importorskip("torch")
    _, n, s, d = case
    want = oracle.cc(oracle.CpuGraph(n, s, d, mirror=True))
    if not device:
        assert np.array_equal(ctx.wcc_edges(n, s, d), want)
        return
    ds, dd = torch.from_numpy(s).cuda(), torch.from_numpy(d).cuda()
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx.wcc_edges(n, (ds.data_ptr(), s.size), (dd.data_ptr(), d.size), out.data_ptr())
    assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("bad", [-1, 7000])
def test_bad_ids_are_refused(ctx, bad):
    s = np.zeros(10, np.int32)
    d = np.arange(10, dtype=np.int32)
    for a, b in ((s, np.where(d == 9, bad, d).astype(np.int32)),
                 (np.where(d == 4, bad, s).astype(np.int32), d)):
        with pytest.raises(gb.GBError) as e:
            ctx.wcc_edges(7000, a, b)
        assert e.value.status == 1  # GB_ERR_INVALID
    assert np.array_equal(ctx.wcc_edges(7000, s, d)[:10], np.zeros(10))


def test_step_cap_keeps_the_searches(ctx):
    n, s, d = graphs.path(10000)
    g = gb.Graph.from_edges(ctx, n, s, d)
    with pytest.raises(gb.GBError) as e:
        ctx.wcc(g, o=gb.opts(max_steps=2))
    assert e.value.status == 5  # GB_ERR_ITER_LIMIT
    with pytest.raises(gb.GBError) as e:
        ctx.wcc_edges(n, s, d, o=gb.opts(max_steps=2))
    assert e.value.status == 5
    assert np.array_equal(ctx.wcc(g), np.zeros(n))
    g.close()
