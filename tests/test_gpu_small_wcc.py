"""WCC of short edge lists in one block: lists that take one, two and several
rounds of hooking, against the oracle, from host and device memory."""
from __future__ import annotations

import numpy as np
import pytest

import connectivity_gb300 as gb
import oracle
from tests import graphs

pytestmark = pytest.mark.gpu


def _relay(k):
    """Stars whose centre has the largest id, chained through their largest
    leaves: leaves of a star meet only after its centre has hooked."""
    leaf = np.arange(10 * k).reshape(k, 10)
    mid = 10 * k + np.arange(k)
    s = np.r_[np.repeat(mid, 10), leaf[:-1, 9]]
    d = np.r_[leaf.ravel(), leaf[1:, 8]]
    return 11 * k, s.astype(np.int32), d.astype(np.int32)


def _perm(n, s, d, seed):
    p = np.random.default_rng(seed).permutation(n).astype(np.int32)
    return n, p[s], p[d]


CASES = {"empty": (70, np.zeros(0, np.int32), np.zeros(0, np.int32)),
         "loops": (9, np.arange(9, dtype=np.int32), np.arange(9, dtype=np.int32)),
         "path": graphs.path(6144), "path_perm": _perm(*graphs.path(6144), 1),
         "cycle_perm": _perm(*graphs.cycle(5000), 2), "relay": _relay(500),
         "relay_perm": _perm(*_relay(558), 3), "grid_perm": _perm(*graphs.grid(70), 4),
         "dense": graphs.erdos(1000, 65536, 5), "sparse": graphs.erdos(6144, 4000, 6)}


@pytest.mark.parametrize("name", CASES)
def test_labels_equal(ctx, name):
    torch = pytest.importorskip("torch")
    n, s, d = CASES[name]
    want = oracle.cc(oracle.CpuGraph(n, s, d, mirror=True))
    assert np.array_equal(ctx.wcc_edges(n, s, d), want)
    ds, dd = torch.from_numpy(s).cuda(), torch.from_numpy(d).cuda()
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx.wcc_edges(n, (ds.data_ptr(), s.size), (dd.data_ptr(), d.size), out.data_ptr())
    assert np.array_equal(out.cpu().numpy(), want)
