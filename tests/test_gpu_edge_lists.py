"""SCC from edge lists above the one-block size: the CSR built by ranges
(csr_part.cu) in its 32- and 64-bit pair forms, at the edges of its ranges,
tiles and chunks, on skewed and even lists; labels against the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import connectivity_gb300 as gb
import oracle
from tests import graphs

pytestmark = pytest.mark.gpu


def _shuffle(n, s, d, seed):
    p = np.random.default_rng(seed).permutation(s.size)
    return n, s[p], d[p]


def _hub(n, m):
    """A hub that every other edge touches: one range holds most entries."""
    r = np.random.default_rng(n)
    s, d = r.integers(0, n, m), r.integers(0, n, m)
    s[::4] = n - 1
    d[1::4] = n - 1
    return n, s.astype(np.int32), d.astype(np.int32)


CASES = [("rmat_6145",) + _shuffle(*gb.rmat_edges_n(6145, 8, 1), 1),
         ("rmat_17",) + _shuffle(*gb.rmat_edges(17, 16, 3), 2),
         # 512 ranges of 256 vertices, and one more vertex
         ("random_2^17",) + graphs.erdos(1 << 17, 300000, 3),
         ("random_2^17+1",) + graphs.erdos((1 << 17) + 1, 300001, 4),
         # tiles of 8,192 edges and chunks of 16,384 entries
         ("tile", 9000) + graphs.erdos(9000, 8192, 5)[1:],
         ("tile+1", 9000) + graphs.erdos(9000, 8193, 6)[1:],
         ("chunk+1", 7000) + graphs.erdos(7000, 16385, 7)[1:],
         ("hub",) + _hub(20000, 400000),
         # the last 32-bit and the first 64-bit pairs
         ("random_2^21",) + graphs.erdos(1 << 21, 3000000, 8),
         ("random_2^21+1",) + graphs.erdos((1 << 21) + 1, 3000000, 9),
         # the largest ranges, and the radix sorts above them
         ("random_2^23",) + graphs.erdos(1 << 23, 5000000, 10),
         ("random_2^23+1",) + graphs.erdos((1 << 23) + 1, 5000000, 11)]


@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
@pytest.mark.parametrize("device", [False, True], ids=["host", "device"])
def test_labels(ctx, case, device):
    torch = pytest.importorskip("torch")
    _, n, s, d = case
    want = oracle.scc(oracle.CpuGraph(n, s, d))
    if not device:
        assert np.array_equal(ctx.scc_edges(n, s, d), want)
        return
    ds, dd = torch.from_numpy(s).cuda(), torch.from_numpy(d).cuda()
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx.scc_edges(n, (ds.data_ptr(), s.size), (dd.data_ptr(), d.size), out.data_ptr())
    assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("case", graphs.edge_cases(), ids=[c[0] for c in graphs.edge_cases()])
def test_small_lists_off_the_one_block_path(ctx, case):
    _, n, s, d = case
    assert np.array_equal(ctx.scc_edges(n, s, d, o=gb.opts(small_path=0)),
                          oracle.scc(oracle.CpuGraph(n, s, d)))


@pytest.mark.parametrize("bad", [-1, 50000, 2**31 - 1])
@pytest.mark.parametrize("at", [0, 8191, 99999])
def test_bad_ids_are_refused(ctx, bad, at):
    n, s, d = graphs.erdos(50000, 100000, 12)
    for k in range(2):
        a, b = s.copy(), d.copy()
        (a, b)[k][at] = bad
        lab = np.full(n, -9, np.int32)
        with pytest.raises(gb.GBError) as e:
            ctx.scc_edges(n, a, b, lab)
        assert e.value.status == 1  # GB_ERR_INVALID
        assert (lab == -9).all()
    assert np.array_equal(ctx.scc_edges(n, s, d), oracle.scc(oracle.CpuGraph(n, s, d)))
