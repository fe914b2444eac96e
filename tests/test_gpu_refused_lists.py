"""An edge list with an id outside [0, n) is refused and leaves the caller's
labels alone, in host and device memory, below and above the one-block size."""
from __future__ import annotations

import numpy as np
import pytest

import connectivity_gb300 as gb
from tests import graphs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["scc", "wcc"])
@pytest.mark.parametrize("n", [5000, 7000, 300000])
@pytest.mark.parametrize("at", [0, 31, -1])
def test_labels_stay(ctx, kind, n, at):
    torch = pytest.importorskip("torch")
    _, s, d = graphs.erdos(n, 3 * n, n)
    d[at] = n
    run = getattr(ctx, kind + "_edges")
    lab = np.full(n, -9, np.int32)
    with pytest.raises(gb.GBError) as e:
        run(n, s, d, lab)
    assert e.value.status == 1  # GB_ERR_INVALID
    assert (lab == -9).all()
    ds, dd, out = (torch.from_numpy(x).cuda() for x in (s, d, lab))
    torch.cuda.synchronize()
    with pytest.raises(gb.GBError) as e:
        run(n, (ds.data_ptr(), s.size), (dd.data_ptr(), d.size), out.data_ptr())
    assert e.value.status == 1
    assert (out.cpu().numpy() == -9).all()
