"""Extrapolated sweeps of the PageRank solvers: graphs on which one error component dominates (power law),
on which none does (a bipartite grid, whose alternating mode meets the rounding), and on which a long step
is wrong (a path: the ratio of residuals is constant until the residual leaves the graph), vertices without
in- or out-edges, part counts around the chunk size, and the capped runs that keep the plain iterates.

Bounds: the stop test bounds the relative L1 error by the tolerance (1e-7); every value is stored in FP32
(2^-24 relative) and each sweep's gathered residual is rounded to FP32, an error the remaining sweeps
amplify by at most 1/(1-d). So the relative L1 error is at most 1e-7 + 2^-24 (1 + 4/(1-d)).
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _graph(E, name):
    if name == "rmat":
        s, d, _ = E.gen_rmat(12, 16, seed=5)
        return 1 << 12, s, d
    if name == "grid":
        s, d, _ = E.gen_grid(64, 0.0, 0.0, seed=1, wmin=1, wmax=1)
        return 64 * 64, s, d
    if name == "path":
        i = np.arange(999, dtype=np.uint32)
        return 1000, i, i + 1
    if name == "cycle":
        i = np.arange(257, dtype=np.uint32)
        return 257, i, (i + 1) % 257
    if name == "star":  # a hub spanning chunks both ways, and vertices without in-edges
        i = np.arange(1, 2000, dtype=np.uint32)
        return 2100, np.concatenate((i[:1500], np.zeros(1000, np.uint32))), np.concatenate((np.zeros(1500, np.uint32), i[:1000]))
    if name == "loop":
        return 2, np.array([0], np.uint32), np.array([0], np.uint32)
    raise KeyError(name)


NAMES = ["rmat", "grid", "path", "cycle", "star", "loop"]


@pytest.mark.parametrize("damping", [0.0, 0.5, 0.99])  # 0: the default, 0.85
@pytest.mark.parametrize("K", [4, 8, 16])
@pytest.mark.parametrize("name", NAMES)
def test_pagerank_extrapolated(gpu, name, K, damping):
    n, s, d = _graph(gpu, name)
    dd = float(np.float32(damping)) if damping else 0.85
    want, _ = oracle.pagerank(n, s, d, damping=dd)
    bound = 1e-7 + 2.0 ** -24 * (1 + 4 / (1 - dd))
    with gpu.VirtualGraph.build(n, s, d, None, K=K, reverse_only=True) as vg:
        for variant in ("sync_push_td", "async_push_td"):
            x, res = vg.run("pr", variant, pr_damping=damping)
            err = np.abs(x.astype(np.float64) - want).sum() / np.abs(want).sum()
            assert err <= bound, (name, variant, err, bound)


@pytest.mark.parametrize("name", ["rmat", "grid", "star"])
def test_pagerank_capped_runs_keep_the_plain_iterates(gpu, name):
    """max_iterations = k: status ITER_CAP and the k-th Jacobi iterate (FP32 rounding of k sweeps)."""
    n, s, d = _graph(gpu, name)
    deg = np.bincount(s, minlength=n)
    with gpu.VirtualGraph.build(n, s, d, None, K=8, reverse_only=True) as vg:
        for k in (1, 7, 20):
            x, res = vg.run("pr", "sync_push_td", max_iterations=k, check=False)
            assert res["status"] == gpu.ERR_ITER_CAP and res["iterations"] == k
            want = np.full(n, 0.15)
            for _ in range(k):
                want = 0.15 + 0.85 * np.bincount(d, weights=(want / np.maximum(deg, 1))[s], minlength=n)
            err = np.abs(x - want).sum() / want.sum()
            assert err <= 2.0 ** -24 * (1 + 4 / 0.15), (k, err)
