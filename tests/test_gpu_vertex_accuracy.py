"""Every vertex's value, not their norm alone: PageRank on graphs with small components, stars and paths, whose
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
