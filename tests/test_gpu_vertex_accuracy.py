"""Every vertex's value, not their norm alone: PageRank and personalised PageRank on graphs with small components, stars and paths, whose
share of the L1 norm is far below the tolerance.

Plain sweeps leave each vertex within about the tolerance of its own value; a run that takes long steps has to
as well. Allowed: eight times the tolerance (the kernels' own bound) and FP32's share. A part's sum takes up to
log2(16) + 3 roundings of 6e-8, and a residual's rounding travels on through the sweeps (1 / (1 - 0.85) in
all): below 3e-6.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(E, name):
    if name == "path":
        n = 5000
        return n, np.arange(n - 1), np.arange(1, n)
    if name == "grid":
        i = np.arange(64 * 64).reshape(64, 64)
        s, d = np.r_[i[:, :-1].ravel(), i[:-1].ravel()], np.r_[i[:, 1:].ravel(), i[1:].ravel()]
        n = 64 * 64
    else:  # isolated pairs, stars and paths come with R-MAT's low-degree vertices
        scale, ef = name
        n = 1 << scale
        s, d, _ = E.gen_rmat(scale, ef, seed=9)
        s, d = s.astype(np.int64), d.astype(np.int64)
    return n, np.r_[s, d], np.r_[d, s]


def _exact(n, s, d, damping):
    sp = pytest.importorskip("scipy.sparse")
    A = sp.csr_matrix((damping / np.bincount(s, minlength=n).astype(float)[s], (d, s)), (n, n))
    f = x = np.full(n, 1 - damping)
    while np.abs(f).sum() > 1e-16 * x.sum():
        f = A @ f
        x = x + f
    return x


@pytest.mark.parametrize("K", [4, 16])
@pytest.mark.parametrize("name", [(12, 16), (16, 2), (16, 16), "path", "grid"], ids=str)
def test_pagerank_vertex_by_vertex(gpu, name, K):
    n, s, d = _graph(gpu, name)
    want = _exact(n, s, d, 0.85)
    with gpu.VirtualGraph.build(n, s.astype(np.uint32), d.astype(np.uint32), None, K=K, reverse_only=True) as vg:
        for tol in (0.0, 1e-4, 1e-2):  # 0: the default, 1e-7
            x, res = vg.run("pr", "sync_push_td", pr_tolerance=tol)
            assert res["status"] == gpu.OK
            off = np.abs(x.astype(np.float64) - want) / want
            assert off.max() <= 8 * (tol or 1e-7) + 3e-6, (tol, off.max(), res["iterations"])


@pytest.mark.parametrize("C,K", [(1, 8), (5, 4), (32, 16), (64, 8)])
@pytest.mark.parametrize("name", [(12, 16), (16, 16)], ids=str)
def test_ppr_element_by_element(gpu, name, C, K):
    """A chunk's row is added up in at most 128 steps and a weight is rounded once per edge of a path: 1e-5."""
    sp = pytest.importorskip("scipy.sparse")
    n, s, d = _graph(gpu, name)
    rng = np.random.default_rng(3)
    w = (rng.random(len(s)) + 0.05).astype(np.float32)
    T = np.zeros((n, C), np.float32)
    for c in range(C):
        T[rng.integers(0, n, 32), c] += 1 / 32
    cols = min(C, 5)
    w64 = w.astype(np.float64)
    A = sp.csr_matrix((0.85 * w64 / np.bincount(s, w64, n)[s], (d, s)), (n, n))
    f = want = 0.15 * T[:, :cols].astype(np.float64)
    while np.abs(f).sum() > 1e-16 * want.sum():
        f = A @ f
        want = want + f
    with gpu.VirtualGraph.build(n, s.astype(np.uint32), d.astype(np.uint32), None, K=K, reverse=True, edge_ids=True) as vg:
        with gpu.PPR(vg, C) as p:
            p.set_weights(w)
            for tol in (0.0, 1e-4):
                x, _ = p.forward(T, tol=tol)
                x = x[:, :cols].astype(np.float64)
                assert np.array_equal(x == 0, want == 0)
                off = (np.abs(x - want)[want > 0] / want[want > 0]).max()
                assert off <= 8 * (tol or 1e-7) + 1e-5, (tol, off)


@pytest.mark.parametrize("C,K", [(1, 8), (5, 4), (64, 8)])
def test_ppr_sources_of_both_signs(gpu, C, K):
    """Values that cancel have no size of their own: the solve ends on its norm, in few sweeps."""
    sp = pytest.importorskip("scipy.sparse")
    n = 1 << 13
    s, d, _ = gpu.gen_rmat(13, 16, seed=2)
    rng = np.random.default_rng(3)
    w = (rng.random(len(s)) + 0.05).astype(np.float32)
    T = rng.standard_normal((n, C)).astype(np.float32)
    A = sp.csr_matrix((0.85 * w.astype(np.float64) / np.bincount(s, w.astype(np.float64), n)[s], (d, s)), (n, n))
    f = want = 0.15 * T.astype(np.float64)
    while np.abs(f).sum() > 1e-16 * np.abs(want).sum():
        f = A @ f
        want = want + f
    with gpu.VirtualGraph.build(n, s, d, None, K=K, reverse=True, edge_ids=True) as vg, gpu.PPR(vg, C) as p:
        p.set_weights(w)
        x, res = p.forward(T)
        assert res["iterations"] < 60, res["iterations"]
        # the tolerance, and FP32's share as in the elements' test; rows of mixed signs cancel to a quarter at worst here
        assert np.abs(x - want).sum() <= (1e-7 + 1e-5) * np.abs(want).sum()
