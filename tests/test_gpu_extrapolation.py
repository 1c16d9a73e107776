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


@pytest.mark.parametrize("damping", [0.0, 0.5, 0.99])
@pytest.mark.parametrize("K", [4, 8, 16])
@pytest.mark.parametrize("name", NAMES)
def test_pagerank_dd_extrapolated(gpu, name, K, damping):
    """Data-driven: FP64 residuals all end at most tol (1-d)^2, so the relative L1 error is at most tol
    (every value is at least 1-d), plus the FP32 rounding of the output."""
    n, s, d = _graph(gpu, name)
    dd = float(np.float32(damping)) if damping else 0.85
    want, _ = oracle.pagerank(n, s, d, damping=dd)
    with gpu.VirtualGraph.build(n, s, d, None, K=K) as vg:
        for variant in ("sync_push_dd", "async_push_dd"):
            x, res = vg.run("pr", variant, pr_damping=damping)
            err = np.abs(x.astype(np.float64) - want).sum() / np.abs(want).sum()
            assert err <= 1e-7 + 2.0 ** -24, (name, variant, err)
            assert res["pr_residual"] <= n * 1e-7 * (1 - dd) ** 2 * 1.0001


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


@pytest.mark.parametrize("C", [1, 5, 32, 64])
@pytest.mark.parametrize("K", [4, 8, 16])
@pytest.mark.parametrize("name", NAMES)
def test_ppr_extrapolated(gpu, name, K, C):
    """Forward and adjoint in residual form against the 64-bit oracle, in the norm of the solve's own bound
    (L1 over all columns). The adjoint's rows, not its columns, sum to at most 1, so its L1 error may exceed
    the bound by the condition of the L1 norm: it is compared in the maximum norm, where the tolerance holds
    up to the norms' ratio on the residual (at most the number of entries), reached on none of these graphs:
    1e-5 of the largest entry."""
    n, s, d = _graph(gpu, name)
    rng = np.random.default_rng(3)
    w = rng.uniform(0.1, 1, s.size).astype(np.float32)
    T = rng.uniform(0, 1, (n, C)).astype(np.float32)
    G = rng.standard_normal((n, C)).astype(np.float32)
    X_ref, _ = oracle.ppr_solve(n, s, d, w, T)
    L_ref, _ = oracle.ppr_solve(n, s, d, w, G, transpose=True)
    with gpu.VirtualGraph.build(n, s, d, None, K=K, reverse=True, edge_ids=True) as vg, gpu.PPR(vg, C) as p:
        p.set_weights(w)
        X, _ = p.forward(T)
        out, _ = p.adjoint(G)
        again, _ = p.adjoint(G)  # the forward's solution survives an adjoint solve
        assert np.array_equal(out["dt"], again["dt"]) and np.array_equal(out["dw"], again["dw"])
    # FP32 weights normalised in FP32 (relative 2^-23), long row sums (star: up to 1500 terms, each addition
    # 2^-24 of the running sum, of random sign: a factor of 8 covers sqrt(1500) / 5), amplified by 1/(1-d)
    bound = 1e-7 + 8 * 2.0 ** -24 / 0.15
    assert np.abs(X - X_ref).sum() <= bound * np.abs(X_ref).sum()
    assert np.abs(out["dt"] - 0.15 * L_ref).max() <= 1e-5 * np.abs(0.15 * L_ref).max()


def test_ppr_capped_runs_keep_the_plain_iterates(gpu):
    n, s, d = _graph(gpu, "rmat")
    rng = np.random.default_rng(4)
    w = rng.uniform(0.1, 1, s.size).astype(np.float32)
    T = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    wn = w / np.bincount(s, weights=w, minlength=n)[s]
    with gpu.VirtualGraph.build(n, s, d, None, K=8, reverse=True, edge_ids=True) as vg, gpu.PPR(vg, 3) as p:
        p.set_weights(w)
        for k in (1, 6):
            X, res = p.forward(T, max_iterations=k, check=False)
            assert res["status"] == gpu.ERR_ITER_CAP and res["iterations"] == k
            want = 0.15 * T.astype(np.float64)
            for _ in range(k):
                want = 0.15 * T + 0.85 * np.stack([np.bincount(d, weights=wn * want[s, c], minlength=n) for c in range(3)], 1)
            assert np.abs(X - want).sum() <= 8 * 2.0 ** -24 / 0.15 * want.sum()


@pytest.mark.parametrize("K", [4, 8, 16])
@pytest.mark.parametrize("hot", [1, 15, 16, 17, 31, 32, 33, 5000])
def test_pagerank_dd_hot_targets(gpu, hot, K):
    """Vertices with more than 64 in-edges (here: 70, `hot` of them, anywhere) collect their pushes in 32 places
    each. The counts lie around a line of places (16), around a warp's vertices (32), and far above. With a
    threshold the rounds stop at |r|_1 / (1-d) of the fixed point; without one, as above."""
    rng = np.random.default_rng(hot)
    n = 20011
    hubs = rng.permutation(n)[:hot]
    s = np.concatenate((rng.integers(0, n, 70 * hot), rng.integers(0, n, 2 * n))).astype(np.uint32)
    d = np.concatenate((np.repeat(hubs, 70), np.repeat(np.arange(n), 2))).astype(np.uint32)
    dd = 0.85
    want, _ = oracle.pagerank(n, s, d, damping=dd)
    with gpu.VirtualGraph.build(n, s, d, None, K=K) as vg:
        for variant, acc in (("sync_push_dd", 0.0), ("async_push_dd", 0.0), ("sync_push_dd", 1e-4), ("sync_push_dd", 1e-7)):
            x, res = vg.run("pr", variant, pr_accuracy=acc)
            err = np.abs(x.astype(np.float64) - want).sum()
            # 2^-24: the output's rounding; 1e-9: the oracle's own stop and the FP64 sums
            bound = res["pr_residual"] / (1 - dd) + (2.0 ** -24 + 1e-9) * np.abs(want).sum()
            assert err <= bound, (variant, acc, err, bound)
            assert acc > 0 or res["pr_residual"] <= n * 1e-7 * (1 - dd) ** 2 * 1.0001
