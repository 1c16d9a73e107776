"""Performance cases: what users of the library have it do, through its public Python entry points.

Every case is a dict of plain values. ``prepare`` makes what a program holds before the call (a graph
resident on the GPU, a batch, a personalised-PageRank handle, or just an edge list), ``run`` makes one
pass, ``work`` states the bytes and operations a pass cannot do without, and ``exact`` gives the
computed (floating-point) outputs in 64 bits. Graphs are R-MAT (0.57/0.19/0.19/0.05, the power-law
graphs of the benchmark; any vertex count, the ids scaled onto it) and the road-like 2-D grid with
shortcuts.

Kinds:
  traverse   BFS / SSSP / SSWP / CC on a resident graph, result left on the GPU
  pagerank   PageRank on a resident graph
  load       an edge list to a result: build, one run, result back in host memory
  batch      many queries over many graphs of uneven size in one launch
  ppr        one step of learning on personalised PageRank: new edge weights, forward, adjoint, gradients
"""
from __future__ import annotations

import math

import numpy as np
import torch

import eegraph_gb300 as E

DEV = "cuda"


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest configured query: one shortest-path query on a 1 M-edge graph, where the launch, the
        # rounds' barriers and the call's own overhead count
        _traverse("sssp_rmat16", "sssp", 1 << 16, 16),
        # the benchmark's 67 M-edge power-law graph: hop counts (with the transposed parts, so that the
        # large rounds may pull) and shortest paths from the hub
        _traverse("bfs_rmat22", "bfs", 1 << 22, 16, reverse=True),
        _traverse("sssp_rmat22", "sssp", 1 << 22, 16),
        # an ordinary graph of no special size, with the larger part size: widest paths from any vertex
        _traverse("sswp_odd_k16", "sswp", 777_777, 23, K=16, source="random"),
        # labels of an undirected graph, every vertex seeded (the reference's ASYNC_PUSH_DD)
        _traverse("cc_sym_rmat21", "cc", 1 << 21, 16, variant="async_push_dd", symmetrize=True),
        # high-diameter road-like graphs: many small rounds. Hop counts on an odd side, and the full
        # 4096 x 4096 configuration's shortest paths with bucketed rounds
        _traverse("bfs_grid2047", "bfs", 2047 * 2047, 0, graph="grid", source="first"),
        _traverse("sssp_grid4096", "sssp", 4096 * 4096, 0, graph="grid", source="first", delta=8000),
        # the benchmark's PageRank (pull sweeps to a relative L1 bound of 1e-7), transposed graph with K = 16
        _pagerank("pr_rmat22", 1 << 22, 16),
        # the reference's residual-push PageRank on a mid-size graph
        _pagerank("pr_dd_rmat17", 1 << 17, 16, variant="sync_push_dd", K=8),
        # a page-locked edge list to distances in host memory: what a one-off query costs
        _load("load_sssp_rmat21", "sssp", 1 << 21, 16, where="host"),
        # many queries over graphs of very different sizes, one launch
        {"name": "batch_64graphs", "kind": "batch", "graphs": 64, "lo": 1 << 10, "hi": 1 << 18, "sources": 8,
         "K": 8},
        # a training step: 64 teleport vectors, gradients of the edge weights and of the teleport vectors
        _ppr("ppr_step_rmat18", 1 << 18, 16, 64),
    ]


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    kind = rng.choice(("rmat", "rmat", "rmat", "grid", "pagerank", "pagerank_dd", "load", "batch", "ppr"))
    K = rng.choice((4, 8, 8, 16))
    if kind == "rmat":
        algo = rng.choice(("bfs", "sssp", "sswp", "cc"))
        n, ef = _log_int(rng, 1 << 16, 1 << 21), rng.randint(8, 32)
        variant = "async_push_dd" if algo == "cc" else rng.choice(("sync_push_dd",) * 3 + ("async_push_dd", "sync_push_td"))
        return _traverse(None, algo, n, ef, K=K, variant=variant, source=rng.choice(("hub", "random")),
                         reverse=algo == "bfs" and rng.random() < 0.5, symmetrize=algo == "cc" or rng.random() < 0.2)
    if kind == "grid":
        algo, delta = rng.choice((("bfs", 0), ("sssp", 8000), ("sssp", 2000), ("sswp", 16), ("sssp", 0)))
        side = _log_int(rng, 256, 2048)
        return _traverse(None, algo, side * side, 0, K=rng.choice((4, 8)), graph="grid", source="first", delta=delta)
    if kind == "pagerank":
        return _pagerank(None, _log_int(rng, 1 << 14, 1 << 21), rng.randint(8, 32), K=K,
                         variant=rng.choice(("sync_push_td",) * 3 + ("async_push_td",)), symmetrize=rng.random() < 0.3)
    if kind == "pagerank_dd":
        return _pagerank(None, _log_int(rng, 1 << 13, 1 << 17), rng.randint(8, 16), K=K,
                         variant=rng.choice(("sync_push_dd", "async_push_dd")))
    if kind == "load":
        algo = rng.choice(("bfs", "sssp", "cc", "pr"))
        return _load(None, algo, _log_int(rng, 1 << 15, 1 << 21), rng.randint(8, 16), K=K,
                     where=rng.choice(("host", "device")))
    if kind == "batch":
        return {"kind": "batch", "graphs": rng.randint(8, 64), "lo": 1 << 10, "hi": _log_int(rng, 1 << 14, 1 << 18),
                "sources": rng.randint(1, 8), "K": rng.choice((8, 8, 16))}
    return _ppr(None, _log_int(rng, 1 << 13, 1 << 18), rng.randint(8, 16), rng.choice((1, 5, 16, 32, 33, 64, 64)), K=K)


def _named(name, case):
    return case if name is None else {"name": name, **case}


def _traverse(name, algo, n, ef, *, K=8, variant="sync_push_dd", graph="rmat", source="hub", reverse=False,
              symmetrize=False, delta=0):
    return _named(name, {"kind": "traverse", "algo": algo, "graph": graph, "n": n, "ef": ef, "K": K, "variant": variant,
                         "source": source, "reverse": reverse, "symmetrize": symmetrize, "delta": delta})


def _pagerank(name, n, ef, *, K=16, variant="sync_push_td", symmetrize=False):
    return _named(name, {"kind": "pagerank", "n": n, "ef": ef, "K": K, "variant": variant, "symmetrize": symmetrize})


def _load(name, algo, n, ef, *, K=8, where="host"):
    return _named(name, {"kind": "load", "algo": algo, "n": n, "ef": ef, "K": K, "where": where})


def _ppr(name, n, ef, columns, *, K=8):
    return _named(name, {"kind": "ppr", "n": n, "ef": ef, "K": K, "columns": columns})


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# ---------------------------------------------------------------- inputs
def _rng(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _rmat(n, ef, gen):
    """Source and target ids (int32) of n * ef R-MAT edges, scaled from the enclosing power of two onto n."""
    scale = max(1, (n - 1).bit_length())
    m = n * ef
    s = torch.zeros(m, dtype=torch.int32, device=DEV)
    d = torch.zeros(m, dtype=torch.int32, device=DEV)
    for _ in range(scale):
        r = torch.rand(m, generator=gen, device=DEV)
        s = (s << 1) + (r >= 0.76).int()
        d = (d << 1) + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95)).int()
    if n != 1 << scale:
        s = ((s.long() * n) >> scale).int()
        d = ((d.long() * n) >> scale).int()
    return s, d


def _grid(side, gen):
    """Arcs (both directions) of a side x side 4-neighbour grid, 10 % of its edges deleted, 0.1 % shortcuts."""
    ids = torch.arange(side * side, dtype=torch.int32, device=DEV).view(side, side)
    a = torch.cat((ids[:, :-1].reshape(-1), ids[:-1, :].reshape(-1)))
    b = torch.cat((ids[:, 1:].reshape(-1), ids[1:, :].reshape(-1)))
    keep = torch.rand(a.numel(), generator=gen, device=DEV) >= 0.1
    cuts = max(1, a.numel() // 1000)
    a, b = a[keep], b[keep]
    a = torch.cat((a, torch.randint(side * side, (cuts,), generator=gen, device=DEV).int()))
    b = torch.cat((b, torch.randint(side * side, (cuts,), generator=gen, device=DEV).int()))
    w = torch.randint(1, 1001, (a.numel(),), generator=gen, device=DEV, dtype=torch.int32)
    return torch.cat((a, b)), torch.cat((b, a)), torch.cat((w, w))


def _weights(m, gen):
    return torch.randint(1, 64, (m,), generator=gen, device=DEV, dtype=torch.int32)


def _edges(case, gen):
    if case.get("graph") == "grid":
        return _grid(math.isqrt(case["n"]), gen)
    s, d = _rmat(case["n"], case["ef"], gen)
    return s, d, _weights(s.numel(), gen)


def _build(n, s, d, w, **kw):
    torch.cuda.synchronize()
    return E.VirtualGraph.build_device(n, s.numel(), s.data_ptr(), d.data_ptr(), None if w is None else w.data_ptr(), **kw)


def _pick_source(case, s, gen):
    if case.get("source") == "first":
        return 0
    if case.get("source") == "random":  # the source of a random edge: a vertex with out-edges
        return int(s[int(torch.randint(s.numel(), (1,), generator=gen, device=DEV))])
    return int(torch.bincount(s).argmax())


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, _rng(seed))


def _prepare_traverse(case, gen):
    s, d, w = _edges(case, gen)
    vg = _build(case["n"], s, d, w, K=case["K"], reverse=case["reverse"], symmetrize=case["symmetrize"])
    return {"run": _run_traverse, "vg": vg, "source": _pick_source(case, s, gen), "algo": case["algo"],
            "variant": case["variant"], "delta": case["delta"],
            "out": torch.empty(case["n"], dtype=torch.int32, device=DEV)}


def _prepare_pagerank(case, gen):
    s, d = _rmat(case["n"], case["ef"], gen)
    dd = case["variant"].endswith("_dd")
    vg = _build(case["n"], s, d, None, K=case["K"], reverse_only=not dd and not case["symmetrize"],
                symmetrize=case["symmetrize"])
    return {"run": _run_pagerank, "vg": vg, "variant": case["variant"],
            "out": torch.empty(case["n"], dtype=torch.float32, device=DEV)}


def _prepare_load(case, gen):
    s, d, w = _edges(case, gen)
    source = _pick_source(case, s, gen)
    edges = [s, d, w]
    if case["where"] == "host":
        edges = [t.cpu().pin_memory().numpy().view(np.uint32) for t in edges]
    out = torch.empty(case["n"], dtype=torch.float32 if case["algo"] == "pr" else torch.int32, pin_memory=True).numpy()
    return {"run": _run_load, "case": case, "edges": edges, "source": source,
            "out": out if case["algo"] == "pr" else out.view(np.uint32)}


def _batch_shapes(case):
    """(vertices, edge factor, queries) per graph: counts spread over [lo, hi] by their logarithm."""
    k, lo, hi = case["graphs"], math.log(case["lo"]), math.log(case["hi"])
    return [(int(round(math.exp(lo + (i + 0.5) / k * (hi - lo)))), 8 + i * 7 % 25, 1 + i * 5 % case["sources"])
            for i in range(k)]


def _prepare_batch(case, gen):
    graphs, queries = [], []
    for i, (n, ef, count) in enumerate(_batch_shapes(case)):
        s, d = _rmat(n, ef, gen)
        graphs.append(_build(n, s, d, _weights(s.numel(), gen), K=case["K"]))
        sources = s[torch.randint(s.numel(), (count,), generator=gen, device=DEV)].cpu().tolist()
        queries += [(i, ("bfs", "sssp", "sswp")[(i + j) % 3], v) for j, v in enumerate(sources)]
    b = E.Batch(graphs)
    words = b.set_queries(queries)
    return {"run": _run_batch, "batch": b, "out": torch.empty(words, dtype=torch.int32, device=DEV)}


def _ppr_inputs(case, gen):
    n, C = case["n"], case["columns"]
    s, d = _rmat(n, case["ef"], gen)
    w = 1.0 - torch.rand(s.numel(), generator=gen, device=DEV)  # (0, 1]
    t = torch.zeros(n, C, device=DEV)
    seeds = torch.randint(n, (32, C), generator=gen, device=DEV)
    t.scatter_add_(0, seeds, torch.full((32, C), 1.0 / 32, device=DEV))  # teleport: uniform over 32 seed vertices
    g = torch.randn(n, C, generator=gen, device=DEV)  # the loss is linear in X
    return s, d, w, t, g


def _prepare_ppr(case, gen):
    s, d, w, t, g = _ppr_inputs(case, gen)
    vg = _build(case["n"], s, d, None, K=case["K"], reverse=True, edge_ids=True)
    return {"run": _run_ppr, "ppr": E.PPR(vg, case["columns"]), "w": w, "t": t, "g": g, "x": torch.empty_like(t),
            "dw": torch.empty_like(w), "dt": torch.empty_like(t)}


# ---------------------------------------------------------------- one pass
def run(state):
    return state["run"](state)


def _run_traverse(st):
    st["vg"].run(st["algo"], st["variant"], st["source"], out_device_ptr=st["out"].data_ptr(), delta=st["delta"])
    return st["out"]


def _run_pagerank(st):
    st["vg"].run("pr", st["variant"], out_device_ptr=st["out"].data_ptr())
    return st["out"]


def _run_load(st):
    case = st["case"]
    s, d, w = st["edges"]
    algo = case["algo"]
    kw = {"K": case["K"], "symmetrize": algo == "cc", "reverse_only": algo == "pr"}
    if algo in ("bfs", "pr"):
        w = None
    if case["where"] == "host":
        vg = E.VirtualGraph.build(case["n"], s, d, w, **kw)
    else:
        vg = E.VirtualGraph.build_device(case["n"], s.numel(), s.data_ptr(), d.data_ptr(),
                                         None if w is None else w.data_ptr(), **kw)
    with vg:
        variant = {"cc": "async_push_dd", "pr": "sync_push_td"}.get(algo, "sync_push_dd")
        vals, _ = vg.run(algo, variant, st["source"], out=st["out"])
    return vals


def _run_batch(st):
    st["batch"].run(st["out"].data_ptr())
    return st["out"]


def _run_ppr(st):
    p = st["ppr"]
    p.set_weights(st["w"].data_ptr())
    p.forward(st["t"].data_ptr(), x_out=st["x"].data_ptr())
    p.adjoint(st["g"].data_ptr(), out_ptrs={"dw": st["dw"].data_ptr(), "dt": st["dt"].data_ptr()})
    return {"x": st["x"], "dw": st["dw"], "dt": st["dt"]}


# ---------------------------------------------------------------- necessary work
def work(case):
    """Each input array read once and each output written once; one relaxation or multiply-add per edge."""
    kind = case["kind"]
    if kind == "batch":
        shapes = _batch_shapes(case)
        return {"bytes": sum(8 * n * ef + q * 4 * n for n, ef, q in shapes), "flops": sum(q * n * ef for n, ef, q in shapes)}
    n = case["n"]
    m = 4 * n * 0.9 if case.get("graph") == "grid" else n * case["ef"]
    if kind == "traverse":
        arcs = 2 * m if case["symmetrize"] else m
        return {"bytes": arcs * (4 if case["algo"] == "bfs" else 8) + 8 * n, "flops": arcs}
    if kind == "pagerank":
        arcs = 2 * m if case["symmetrize"] else m
        return {"bytes": arcs * 4 + 12 * n, "flops": 2 * arcs}
    if kind == "load":  # the edge list in, the result out
        return {"bytes": m * (8 if case["algo"] in ("bfs", "pr") else 12) + 4 * n, "flops": m}
    # weights, both ids and the weight gradient per edge; teleport, dLoss/dX, X and dLoss/dT rows
    return {"bytes": 16 * m + 16 * n * case["columns"], "flops": 6 * m * case["columns"]}


# ---------------------------------------------------------------- 64-bit results
def exact(case, seed):
    """PageRank and personalised PageRank with its gradients in 64 bits; None where outputs are whole numbers."""
    gen = _rng(seed)
    if case["kind"] == "pagerank":
        s, d = _rmat(case["n"], case["ef"], gen)
        if case["symmetrize"]:
            s, d = torch.cat((s, d)), torch.cat((d, s))
        return _exact_pagerank(case["n"], s, d)
    if case["kind"] == "load" and case["algo"] == "pr":
        s, d, _ = _edges(case, gen)
        return _exact_pagerank(case["n"], s, d).cpu().numpy()
    if case["kind"] == "ppr":
        return _exact_ppr(case, *_ppr_inputs(case, gen))
    return None


def _csr(n, rows, cols, vals):
    order = torch.argsort(rows, stable=True)
    crow = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    crow[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    return torch.sparse_csr_tensor(crow, cols[order].long(), vals[order], size=(n, n))


def _solve(A, b, d=0.85, tol=1e-15):
    """x = b + d A x by plain iteration, A with row or column sums at most 1."""
    x = b
    for _ in range(400):
        y = b + d * (A @ x)
        done = float((y - x).abs().sum()) <= tol * float(y.abs().sum())
        x = y
        if done:
            break
    return x


def _exact_pagerank(n, s, d):
    deg = torch.bincount(s, minlength=n).double()
    A = _csr(n, d, s, (1.0 / deg)[s.long()])
    return _solve(A, torch.full((n,), 0.15, dtype=torch.float64, device=DEV))


def _exact_ppr(case, s, d, w, t, g):
    n = case["n"]
    s, d, w, t, g = s.long(), d.long(), w.double(), t.double(), g.double()
    out = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, s, w)
    wn = w / out[s]
    X = _solve(_csr(n, d, s, wn), 0.15 * t)
    L = _solve(_csr(n, s, d, wn), g)
    gw = torch.cat([0.85 * (X[a] * L[b]).sum(1) for a, b in zip(s.split(1 << 20), d.split(1 << 20))])
    r = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, s, gw * wn)
    return {"x": X, "dw": (gw - r[s]) / out[s], "dt": 0.15 * L}
