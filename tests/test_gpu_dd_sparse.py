"""Data-driven PageRank on both sides of the line (a part per four vertices) below which its rounds keep a queue instead
of taking long steps: every vertex within the run's own bound, residuals at most tol (1-d)^2, of its value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sources", [9_999, 10_000, 300])  # of 40000 vertices, one part each
@pytest.mark.parametrize("K", [4, 16])
def test_queue_and_long_steps(gpu, sources, K):
    sp = pytest.importorskip("scipy.sparse")
    n = 40_000
    rng = np.random.default_rng(sources)
    s = np.repeat(np.arange(sources), 3)
    d = np.concatenate((rng.integers(0, sources, sources)[:, None], rng.integers(0, n, (sources, 2))), axis=1).ravel()
    with gpu.VirtualGraph.build(n, s.astype(np.uint32), d.astype(np.uint32), None, K=K) as vg:
        assert vg.info()["num_parts"] == sources
        x, res = vg.run("pr", "sync_push_dd")
    assert res["status"] == gpu.OK
    A = sp.csr_matrix((np.full(s.size, 0.85 / 3), (d, s)), (n, n))
    want = f = np.full(n, 0.15)
    while (f / want).max() > 1e-15:
        f = A @ f
        want = want + f
    # ||x* - x||_1 <= ||r||_1 / (1-d) <= n tol (1-d); the output is FP32
    assert np.abs(x - want).sum() <= n * 1e-7 * 0.15 + 6e-8 * want.sum()
