"""The workloads that this framework's speed is measured on.

A case is one call as a user's program makes it, over one of the graph
families of this repository (seeded R-MAT graphs, oriented lattices with
chains, log-normal batches of R-MAT graphs):

  scc, wcc              Context.scc / wcc on a device-resident graph, labels
                        into a device buffer
  scc_edges, wcc_edges  Context.scc_edges / wcc_edges: an edge list (host
                        arrays, or device buffers) to labels in one call
  run_scc, run_cc       the drop-ins with the reference's signature: its
                        32-bit CSR in host memory in, host labels out
  batch_scc, batch_wcc  many independent graphs as one resident union
  serve                 a burst of requests through the server, host edges
                        in, host labels out

Every output is an array of int32 component labels.
"""
from __future__ import annotations

import numpy as np
import torch

import connectivity_gb300 as gb


def listed() -> list[dict]:
    return [
        # One small request from an edge list in host memory: the smallest
        # call, where the launch and the copies count.
        {"name": "edges_scc_300", "op": "scc_edges", "n": 300, "ef": 8, "device": False,
         "shuffled": False},
        # A small resident graph analysed on its own.
        {"name": "scc_4000", "op": "scc", "family": "rmat", "n": 4000, "ef": 16},
        # The small benchmark graph (R-MAT scale 16): a mid-size resident
        # graph, bound by its steps and not by its bytes.
        {"name": "scc_rmat16", "op": "scc", "family": "rmat", "n": 1 << 16, "ef": 16},
        # The headline benchmark: SCC of R-MAT scale 24.
        {"name": "scc_rmat24", "op": "scc", "family": "rmat", "n": 1 << 24, "ef": 16},
        # Weak components of a directed graph of odd size.
        {"name": "wcc_rmat_3m", "op": "wcc", "family": "rmat", "n": 3_000_017, "ef": 16},
        # The high-diameter benchmark family: SCC (long propagations) ...
        {"name": "scc_grid1024", "op": "scc", "family": "grid", "side": 1024},
        # ... and its weak components.
        {"name": "wcc_grid2048", "op": "wcc", "family": "grid", "side": 2048},
        # The reference's program with one call swapped: its own malloc'd
        # CSR arrays, end to end.
        {"name": "run_scc_rmat22", "op": "run_scc", "n": 1 << 22, "ef": 16, "pinned": False},
        # The same for cc, from a caller that pins its buffers.
        {"name": "run_cc_rmat22", "op": "run_cc", "n": 1 << 22, "ef": 16, "pinned": True},
        # An edge list already on the device, in generator order, to labels:
        # the CSR build and the run together.
        {"name": "edges_scc_rmat20", "op": "scc_edges", "n": 1 << 20, "ef": 16, "device": True,
         "shuffled": True},
        # Many independent graphs at once (the batched benchmark's sizes).
        {"name": "batch_scc_2000", "op": "batch_scc", "count": 2000},
        # A burst of requests (the served benchmark's mix, all at once).
        {"name": "serve_1000", "op": "serve", "requests": 1000, "pool": 64},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    v = int(round(lo * (hi / lo) ** rng.random()))
    return max(lo, min(hi, v))


def _rmat_size(rng, lo: int, hi: int, edges: int) -> tuple[int, int]:
    """A vertex count in [lo, hi] and an edge factor in 4..32, at most
    `edges` candidate edges."""
    n = _log_int(rng, lo, hi)
    return n, max(4, min(rng.randint(4, 32), edges // n))


def draw(rng) -> dict:
    op = rng.choice(["scc", "wcc", "scc", "wcc", "scc_edges", "wcc_edges", "run_scc", "run_cc",
                     "batch_scc", "batch_wcc", "serve"])
    if op in ("scc", "wcc"):
        if rng.random() < 0.3:
            return {"op": op, "family": "grid",
                    "side": _log_int(rng, 100, 1024 if op == "scc" else 4096)}
        n, ef = _rmat_size(rng, 300, 1 << 24, 1 << 28)
        return {"op": op, "family": "rmat", "n": n, "ef": ef}
    if op in ("scc_edges", "wcc_edges"):
        n, ef = _rmat_size(rng, 64, 1 << 21, 1 << 25)
        return {"op": op, "n": n, "ef": ef, "device": rng.random() < 0.5,
                "shuffled": rng.random() < 0.5}
    if op in ("run_scc", "run_cc"):
        n, ef = _rmat_size(rng, 10_000, 1 << 22, 1 << 26)
        return {"op": op, "n": n, "ef": ef, "pinned": rng.random() < 0.5}
    if op in ("batch_scc", "batch_wcc"):
        return {"op": op, "count": _log_int(rng, 50, 2000)}
    return {"op": op, "requests": _log_int(rng, 100, 1000), "pool": 64}


def _host(count: int, pinned: bool) -> np.ndarray:
    """An int32 host array, malloc'd or pinned."""
    if pinned:
        return torch.empty(count, dtype=torch.int32).pin_memory().numpy()
    return np.empty(count, np.int32)


def _edges(ctx, n: int, ef: int, seed: int, shuffled: bool):
    """Device edge list of an R-MAT graph, sorted by source or in random
    order."""
    g = gb.Graph.rmat_n(ctx, n, ef, seed)
    off, adj, _, _ = g.to_host()
    g.close()
    deg = torch.from_numpy(np.diff(off)).cuda()
    src = torch.repeat_interleave(torch.arange(n, dtype=torch.int32, device="cuda"), deg)
    dst = torch.from_numpy(adj).cuda()
    if shuffled:
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        p = torch.randperm(src.numel(), generator=gen, device="cuda")
        src, dst = src[p], dst[p]
    return src.contiguous(), dst.contiguous()


def _batch(count: int, seed: int):
    """Sizes of the batched benchmark's distribution (the same for every
    seed), and per-graph seeds."""
    ns, efs, seeds = gb.batch_sizes(count)
    return ns, efs, seeds + np.uint64(seed)


def prepare(case: dict, seed: int) -> dict:
    op = case["op"]
    s = {"op": op}
    if op in ("run_scc", "run_cc"):
        ctx = gb.Context(0)
        g = gb.Graph.rmat_n(ctx, case["n"], case["ef"], seed)
        oo, oa, io, ia = g.to_host()
        n = g.n
        g.close()
        if op == "run_cc":  # cc's mirrored graph: every vertex's out- and in-neighbours
            do, di = np.diff(oo), np.diff(io)
            off = oo + io
            adj = np.empty(off[n], np.int32)
            adj[np.arange(oa.size) + np.repeat(io[:-1], do)] = oa
            adj[np.arange(ia.size) + np.repeat(oo[1:], di)] = ia
            oo, oa, io, ia = off, adj, None, None
        for key, a in (("oo", oo), ("oa", oa), ("io", io), ("ia", ia)):
            if a is not None:
                s[key] = _host(a.size, case["pinned"])
                s[key][:] = a
        for key in ("oo", "io"):
            if key in s:
                s[key] = s[key].view(np.uint32)
        s.update(n=n, labels=_host(n, case["pinned"]))
        ctx.close()
    elif op == "serve":
        ns, efs, seeds = _batch(case["pool"], seed)
        pool = []
        for n, ef, gs in zip(ns, efs, seeds):
            _, src, dst = gb.rmat_edges_n(int(n), int(ef), int(gs))
            ps, pd = _host(src.size, True), _host(dst.size, True)
            ps[:], pd[:] = src, dst
            pool.append((int(n), ps, pd))
        r = np.random.default_rng(4)
        pick = r.integers(0, case["pool"], case["requests"])
        kind = (r.random(case["requests"]) < 0.2).astype(int)  # 80 % SCC, 20 % WCC
        base = np.concatenate([[0], np.cumsum([pool[p][0] for p in pick])])
        s["labels"] = _host(int(base[-1]), True)
        s["requests"] = [(int(k), pool[p][0], pool[p][1], pool[p][2], s["labels"][a:b])
                         for k, p, a, b in zip(kind, pick, base[:-1], base[1:])]
        s["ctx"] = gb.Context(0)
        s["server"] = gb.Server(s["ctx"], 8 << 30)
        s["server"].start()
    else:
        ctx = s["ctx"] = gb.Context(0)
        if op in ("scc_edges", "wcc_edges"):
            src, dst = _edges(ctx, case["n"], case["ef"], seed, case["shuffled"])
            s["n"] = case["n"]
            if case["device"]:
                s["keep"] = (src, dst)
                s["src"], s["dst"] = (src.data_ptr(), src.numel()), (dst.data_ptr(), dst.numel())
                s["labels"] = torch.empty(s["n"], dtype=torch.int32, device="cuda")
                s["out"] = s["labels"].data_ptr()
            else:
                s["src"], s["dst"] = src.cpu().numpy(), dst.cpu().numpy()
                s["labels"] = s["out"] = np.empty(s["n"], np.int32)
        else:
            if op in ("batch_scc", "batch_wcc"):
                s["g"] = gb.Batch.rmat(ctx, *_batch(case["count"], seed))
            elif case["family"] == "grid":
                s["g"] = gb.Graph.from_edges(ctx, *gb.grid_edges(case["side"], seed=seed))
            else:
                s["g"] = gb.Graph.rmat_n(ctx, case["n"], case["ef"], seed)
            s["labels"] = torch.empty(s["g"].n, dtype=torch.int32, device="cuda")
            s["out"] = s["labels"].data_ptr()
    torch.cuda.synchronize()
    return s


def run(s: dict):
    op = s["op"]
    if op == "scc":
        s["ctx"].scc(s["g"], s["out"])
    elif op == "wcc":
        s["ctx"].wcc(s["g"], s["out"])
    elif op == "scc_edges":
        s["ctx"].scc_edges(s["n"], s["src"], s["dst"], s["out"])
    elif op == "wcc_edges":
        s["ctx"].wcc_edges(s["n"], s["src"], s["dst"], s["out"])
    elif op == "run_scc":
        gb.run_scc_ref(s["n"], s["oa"], s["ia"], s["oo"], s["io"], scc_maps=s["labels"])
    elif op == "run_cc":
        gb.run_cc_ref(s["n"], s["oa"], s["oo"], cc_maps=s["labels"])
    elif op == "batch_scc":
        s["ctx"].batch_scc(s["g"], s["out"])
    elif op == "batch_wcc":
        s["ctx"].batch_wcc(s["g"], s["out"])
    else:
        srv = s["server"]
        for kind, n, src, dst, out in s["requests"]:
            srv.submit(kind, n, src, dst, out=out)
        srv.drain()
    return s["labels"]


def work(case: dict) -> dict:
    """Every edge once, the vertex offsets once, the labels written once.
    (The in-lists of a resident graph or of run_scc's arrays are the out-lists
    transposed, so one of the two suffices; edge counts are the generators'
    candidates, of which a few per cent are duplicates.)"""
    op = case["op"]
    if op in ("scc", "wcc"):
        if case["family"] == "grid":
            side = case["side"]
            n = side * side + side * side // 10
            m = 2 * side * side + side * side // 10
        else:
            n, m = case["n"], case["n"] * case["ef"]
        return {"bytes": 8 * (n + 1) + 4 * m + 4 * n, "flops": 0}
    if op in ("scc_edges", "wcc_edges"):
        return {"bytes": 8 * case["n"] * case["ef"] + 4 * case["n"], "flops": 0}
    if op in ("run_scc", "run_cc"):
        n, m = case["n"], case["n"] * case["ef"] * (1 if op == "run_scc" else 2)
        return {"bytes": 4 * (n + 1) + 4 * m + 4 * n, "flops": 0}
    # batches and requests: the distribution's mean graph has about 5,900
    # vertices and 18 edges per vertex
    graphs = case["count"] if op in ("batch_scc", "batch_wcc") else case["requests"]
    n, m = 5900 * graphs, 5900 * 18 * graphs
    if op == "serve":
        return {"bytes": 8 * m + 4 * n, "flops": 0}
    return {"bytes": 8 * (n + 1) + 4 * m + 4 * n, "flops": 0}
