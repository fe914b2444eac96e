"""The contraction's buffer: not taken for graphs whose hubs are known, given
back after the run, and done without where the pool refuses it."""
from __future__ import annotations

import contextlib
import ctypes as C

import numpy as np
import pytest

import connectivity_gb300 as gb
import oracle
from tests import graphs

pytestmark = pytest.mark.gpu

ROUND = 22  # trace mode of a contraction round


class _PoolProps(C.Structure):  # CUmemPoolProps
    _fields_ = [("alloc_type", C.c_int), ("handle_types", C.c_int), ("loc_type", C.c_int),
                ("loc_id", C.c_int), ("win32", C.c_void_p), ("max_size", C.c_size_t),
                ("usage", C.c_ushort), ("reserved", C.c_ubyte * 54)]


@contextlib.contextmanager
def _small_pool(max_size):
    """The device's current memory pool is one of at most max_size bytes."""
    cuda = C.CDLL("libcuda.so.1")

    def ok(status):
        assert status == 0, status

    dev, old, pool = C.c_int(), C.c_void_p(), C.c_void_p()
    ok(cuda.cuDeviceGet(C.byref(dev), 0))
    ok(cuda.cuDeviceGetMemPool(C.byref(old), dev))
    props = _PoolProps(alloc_type=1, loc_type=1, loc_id=0, max_size=max_size)
    ok(cuda.cuMemPoolCreate(C.byref(pool), C.byref(props)))
    ok(cuda.cuDeviceSetMemPool(dev, pool))
    try:
        yield
    finally:
        ok(cuda.cuDeviceSetMemPool(dev, old))
        ok(cuda.cuMemPoolDestroy(pool))


def test_runs_without_the_buffer():
    ctx = gb.Context(0)
    n, s, d = graphs.grid(1200)
    g = gb.Graph.from_edges(ctx, n, s, d)  # 48 MB for the contraction (pools grow by 32)
    want = oracle.scc(oracle.CpuGraph(n, s, d))
    assert np.array_equal(ctx.scc(g), want)
    assert ROUND in [r[2] for r in ctx.reach_trace()]
    with _small_pool(2 << 20):
        assert np.array_equal(ctx.scc(g), want)
        assert ROUND not in [r[2] for r in ctx.reach_trace()]
    assert np.array_equal(ctx.scc(g), want)
    assert ROUND in [r[2] for r in ctx.reach_trace()]
    g.close()
    ctx.close()


@pytest.mark.parametrize("hub", [False, True])
def test_buffer_is_not_kept(hub):
    """100 MB of edge pairs: none for an R-MAT graph of 4 edges per vertex,
    whose hubs the hint build has seen, and none held after a lattice's run."""
    torch = pytest.importorskip("torch")
    ctx = gb.Context(0)
    n, s, d = gb.rmat_edges(21, 4, 1) if hub else graphs.grid(1800)
    g = gb.Graph.from_edges(ctx, n, s, d)
    lab = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()

    def free():  # with what the pools hold but do not use
        ctx.sync()
        cuda, pool = C.CDLL("libcuda.so.1"), C.c_void_p()
        assert cuda.cuDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
        assert cuda.cuMemPoolTrimTo(pool, C.c_size_t(0)) == 0
        return torch.cuda.mem_get_info(0)[0]

    ctx.scc(g, lab.data_ptr(), gb.opts(colour_mode=0))  # the workspace
    before = free()
    ctx.scc(g, lab.data_ptr())
    assert before - free() < 16 << 20
    assert np.array_equal(lab.cpu().numpy(), oracle.scc(oracle.CpuGraph(n, s, d)))
    g.close()
    ctx.close()
